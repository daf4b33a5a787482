// row_grid.h -- grids of tiles whose rows may outnumber a grid dimension.
#pragma once

#include <cuda_runtime.h>

namespace zg {

// Grid of `across` x `rows` tiles: a grid's second and third dimension end at
// 65535 blocks, and a tube may have 2^28 rows.  Row tile of a block: blockIdx.z *
// gridDim.y + blockIdx.y; the last ones may lie past `rows`.  (One dimension and
// a division in each thread cost 1.5 % of a PARITY step at 1031 x 517.)
inline dim3 row_grid(unsigned across, unsigned rows) {
    const unsigned layers = (rows + 65534) / 65535;
    return dim3(across, (rows + layers - 1) / layers, layers);
}

}  // namespace zg
