// host_copy.cu -- large copies between device arrays and pageable host memory.
//
// A plain cudaMemcpy to pageable memory runs at 3-4 GB/s on a B200 box where
// the destination is fresh (each page is touched for the first time by one
// thread): 42 MB 10.3 ms, 168 MB 40 ms.  Here four host threads each move
// every fourth chunk through two pinned slots of their own, so that the DMA
// of one chunk, the copies of others into the caller's pages and the page
// faults of those run at the same time.
//
// The pinned memory (8 slots of 2 MB) and the streams belong to the process,
// are made at the first large copy and given back with the last context.  One
// copy at a time uses them; a second one meanwhile, small copies, and arrays
// that are pinned or on a device already, take the plain path.
#include "host_copy.h"

#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

namespace zg {
namespace host {
namespace {

constexpr int THREADS = 4, SLOTS = 2 * THREADS, MAX_DEV = 64;
constexpr size_t CHUNK = size_t(2) << 20;
// below this the threads cost more than they save (a copy of 4 MB takes about 1 ms)
constexpr size_t MIN_BYTES = size_t(4) << 20;

struct Staging {
    std::mutex busy;   // held by the copy that uses the slots
    std::mutex count;  // guards `users`
    int users = 0;
    unsigned char *pinned = nullptr;
    cudaStream_t stream[MAX_DEV][SLOTS] = {};
};
Staging g_staging;

void drop() {  // `busy` held
    if (g_staging.pinned) cudaFreeHost(g_staging.pinned);
    g_staging.pinned = nullptr;
    for (int d = 0; d < MAX_DEV; ++d) {
        if (!g_staging.stream[d][0]) continue;
        int prev = -1;
        cudaGetDevice(&prev);
        cudaSetDevice(d);
        for (cudaStream_t &s : g_staging.stream[d]) {
            if (s) cudaStreamDestroy(s);
            s = nullptr;
        }
        if (prev >= 0) cudaSetDevice(prev);
    }
}

cudaError_t ready(int device) {  // `busy` held; the slots and the device's streams exist
    if (!g_staging.pinned) {
        void *p = nullptr;
        cudaError_t e = cudaHostAlloc(&p, SLOTS * CHUNK, cudaHostAllocPortable);
        if (e != cudaSuccess) return e;
        g_staging.pinned = static_cast<unsigned char *>(p);
    }
    for (cudaStream_t &s : g_staging.stream[device])
        if (!s) {
            cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// Chunk k of the pieces laid end to end, each cut into chunks of its own.
struct Chunks {
    const Piece *pieces;
    int n;
    size_t total;
    bool at(size_t k, unsigned char *&h, unsigned char *&d, size_t &bytes) const {
        for (int p = 0; p < n; ++p) {
            const size_t own = (pieces[p].bytes + CHUNK - 1) / CHUNK;
            if (k < own) {
                const size_t off = k * CHUNK;
                h = static_cast<unsigned char *>(pieces[p].host) + off;
                d = static_cast<unsigned char *>(const_cast<void *>(pieces[p].dev)) + off;
                bytes = pieces[p].bytes - off < CHUNK ? pieces[p].bytes - off : CHUNK;
                return true;
            }
            k -= own;
        }
        return false;
    }
};

// Thread t's share: chunks t, t + THREADS, ... through slots 2 t and 2 t + 1 in
// turn.  A slot's stream has at most one copy in flight.
cudaError_t share(int device, const Chunks &c, int t, bool to_host) {
    cudaError_t e = cudaSetDevice(device);
    unsigned char *dst[2] = {};
    size_t len[2] = {};
    unsigned turn = 0;
    auto finish = [&](unsigned s) {  // wait for the slot; a download's bytes go on to the caller
        const cudaError_t r = cudaStreamSynchronize(g_staging.stream[device][2 * t + s]);
        if (r == cudaSuccess && to_host && len[s])
            std::memcpy(dst[s], g_staging.pinned + (2 * t + s) * CHUNK, len[s]);
        len[s] = 0;
        if (e == cudaSuccess) e = r;
    };
    for (size_t k = t; e == cudaSuccess; k += THREADS, ++turn) {
        unsigned char *h, *d;
        size_t bytes;
        if (!c.at(k, h, d, bytes)) break;
        const unsigned s = turn & 1;
        unsigned char *slot = g_staging.pinned + (2 * t + s) * CHUNK;
        finish(s);
        if (e != cudaSuccess) break;
        if (!to_host) std::memcpy(slot, h, bytes);
        e = to_host ? cudaMemcpyAsync(slot, d, bytes, cudaMemcpyDeviceToHost, g_staging.stream[device][2 * t + s])
                    : cudaMemcpyAsync(d, slot, bytes, cudaMemcpyHostToDevice, g_staging.stream[device][2 * t + s]);
        dst[s] = h;
        len[s] = bytes;
    }
    finish(turn & 1);  // the older slot first
    finish((turn & 1) ^ 1);
    return e;
}

cudaError_t plain(cudaStream_t st, const Piece *p, int n, bool to_host) {
    for (int k = 0; k < n; ++k) {
        cudaError_t e = to_host ? cudaMemcpyAsync(p[k].host, p[k].dev, p[k].bytes, cudaMemcpyDeviceToHost, st)
                                : cudaMemcpyAsync(const_cast<void *>(p[k].dev), p[k].host, p[k].bytes,
                                                  cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(st);
}

}  // namespace

void retain() {
    std::lock_guard<std::mutex> l(g_staging.count);
    ++g_staging.users;
}
void release() {
    std::lock_guard<std::mutex> l(g_staging.count);
    if (--g_staging.users == 0) {
        std::lock_guard<std::mutex> b(g_staging.busy);
        drop();
    }
}

cudaError_t copy(int device, cudaStream_t st, const Piece *pieces, int n, bool to_host) {
    size_t total = 0;
    bool pageable = device >= 0 && device < MAX_DEV;
    for (int k = 0; k < n; ++k) {
        total += pieces[k].bytes;
        cudaPointerAttributes at{};
        if (cudaPointerGetAttributes(&at, pieces[k].host) != cudaSuccess) {
            cudaGetLastError();
            pageable = false;
        } else if (at.type != cudaMemoryTypeUnregistered) {
            pageable = false;
        }
    }
    if (total < MIN_BYTES || !pageable) return plain(st, pieces, n, to_host);
    std::unique_lock<std::mutex> own(g_staging.busy, std::try_to_lock);
    if (!own.owns_lock()) return plain(st, pieces, n, to_host);
    if (ready(device) != cudaSuccess) {
        cudaGetLastError();
        drop();
        return plain(st, pieces, n, to_host);
    }
    cudaError_t e = cudaStreamSynchronize(st);  // the work before the copy
    if (e != cudaSuccess) return e;
    const Chunks c{pieces, n, total};
    cudaError_t got[THREADS] = {};
    std::thread th[THREADS];
    for (int t = 1; t < THREADS; ++t) {
        try {
            th[t] = std::thread([&, t] { got[t] = share(device, c, t, to_host); });
        } catch (const std::system_error &) {  // no thread to be had: its share is done below
        }
    }
    got[0] = share(device, c, 0, to_host);
    for (int t = 1; t < THREADS; ++t) {
        if (th[t].joinable()) th[t].join();
        else got[t] = share(device, c, t, to_host);
    }
    for (cudaError_t x : got)
        if (x != cudaSuccess) return x;
    return cudaSuccess;
}

}  // namespace host
}  // namespace zg
