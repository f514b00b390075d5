// Register-pencil xy passes, double (fft_reg.cuh)
#include "fft_reg.cuh"
#include "fft_reg_api.cuh"

namespace gfix {

template <>
RegXy<double> reg_xy<double>(int n, int per) {
  RegXy<double> r;
#define GFIX_X1(N, PL)                                        \
  if (n == N && per % PL == 0 && !r.fn[0]) {                  \
    r.fn[0] = k_fft_xy_reg<double, N, PL, false>;             \
    r.fn[1] = k_fft_xy_reg<double, N, PL, true>;              \
    r.planes = PL;                                            \
    r.threads = N * PL;                                       \
    r.smem = xy_reg_smem<double, N, PL>();                    \
  }
#define GFIX_P(N, PL)                                         \
  if (n == N && per % PL == 0 && !r.fn[0]) {                  \
    r.fn[0] = k_fft_xy_pair<double, N, PL, false>;            \
    r.fn[1] = k_fft_xy_pair<double, N, PL, true>;             \
    r.planes = PL;                                            \
    r.threads = 2 * N * PL;                                   \
    r.smem = xy_reg_smem<double, N, PL>();                    \
  }
  GFIX_P(36, 4) GFIX_P(40, 2) GFIX_P(48, 1) GFIX_P(64, 1)
#define GFIX_X(N) GFIX_X1(N, (N <= 32 ? 4 : 2)) GFIX_X1(N, 2) GFIX_X1(N, 1)
  GFIX_X(4) GFIX_X(6) GFIX_X(8) GFIX_X(10) GFIX_X(12) GFIX_X(14) GFIX_X(16) GFIX_X(18)
  GFIX_X(20) GFIX_X(24) GFIX_X(28) GFIX_X(30) GFIX_X(32)
#undef GFIX_P
#undef GFIX_X
#undef GFIX_X1
  return r;
}

}  // namespace gfix
