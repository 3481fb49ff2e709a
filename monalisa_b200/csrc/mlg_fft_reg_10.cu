// Register line-FFT passes, group 10 of the axis lengths (mlg_fft_reg_lengths.h).
#include "mlg_fft_reg.cuh"
#include "mlg_fft_reg_lengths.h"

namespace mlg {

int fft_reg_group_10(const FftAxisPlan& a, PassMode mode, const PassDesc& d, int* n_partial, cudaStream_t s,
                    bool* done) {
  switch (a.N) {
#define X(N, A, B, MAIN) \
  case N: return reg_dispatch<A, B, MAIN>(a, mode, d, n_partial, s, done);
    MLG_REG_GROUP_10(X)
#undef X
    default: return MLG_OK;
  }
}

}  // namespace mlg
