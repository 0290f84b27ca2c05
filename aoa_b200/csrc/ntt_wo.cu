// The column passes with warp-owned columns (ntt_kernels.cuh).
#include "ntt_kernels.cuh"

namespace aoa {

void run_cols_wo(const Engine& E, const NttBatch& b, int div, bool fwd, cudaStream_t st) {
  switch (b.log_r * 4 + div) {
#define AOA_WO(s)                                                    \
  case s * 4 + 0: launch_cols_wo<s, 8>(E, b, fwd, st); return;       \
  case s * 4 + 1: launch_cols_wo<s, 4>(E, b, fwd, st); return;       \
  case s * 4 + 2: launch_cols_wo<s, 2>(E, b, fwd, st); return;
    AOA_WO(6) AOA_WO(7) AOA_WO(8) AOA_WO(9)
#undef AOA_WO
    default: throw AoaError(AOA_ERR_BAD_PARAM, "ntt: unsupported column size");
  }
}

template <int S, int NW>
static void allow_wo() {
  allow_smem(ntt_cols_wo<S, NW, true>, WoTile<S, NW>::SMEM);
  allow_smem(ntt_cols_wo<S, NW, false>, WoTile<S, NW>::SMEM);
}

void allow_wo_kernels() {
#define AOA_ALLOW_WO(s) allow_wo<s, 8>(); allow_wo<s, 4>(); allow_wo<s, 2>();
  AOA_ALLOW_WO(6) AOA_ALLOW_WO(7) AOA_ALLOW_WO(8) AOA_ALLOW_WO(9)
#undef AOA_ALLOW_WO
}

}  // namespace aoa
