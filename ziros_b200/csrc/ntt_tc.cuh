// ntt_tc.cuh — Goldilocks NTT passes on the tensor cores (ntt_tc.cu).
#pragma once
#include <cuda.h>

#include "ntt_tile.cuh"

namespace zkb {
namespace ntt_tc {

// Columns of a tile of a K-bit pass, 0 where no such kernel exists.
uint32_t chunk(int K);
// One pass over `tiles` tiles (g.chunks_per_row chunks of `chunk` columns, the last may have fewer); `map`
// describes the input (pass_tensor_map with that chunk), tw the twiddles of the direction.
int pass(int K, uint64_t *out, const PassGeom &g, uint64_t tiles, const uint64_t *tw, bool inverse, uint64_t scale,
         const CUtensorMap &map, cudaStream_t s);
// The fused LDE middle over `tiles` tiles, tables as lde_fused_kernel's.
int fused(int K, uint64_t *out, const FusedGeom &g, uint64_t tiles, const uint64_t *itw, const uint64_t *ftw,
          const uint64_t *ctab_t, const uint64_t *ftw_t, const CUtensorMap &map, cudaStream_t s);

}  // namespace ntt_tc
}  // namespace zkb
