// Register-pencil (z, t) and Coulomb z passes, double (fft_reg.cuh)
#include "fft_reg.cuh"
#include "fft_reg_api.cuh"

namespace gfix {

template <>
RegZt<double> reg_zt<double>(int lz, int lt, int lx, int want) {
  RegZt<double> r;
#define GFIX_T(LZ, LT, B)                                                           \
  if (lz == LZ && lt == LT && lx % B == 0 && (want ? want == B : !r.fn)) {          \
    r.fn = k_fft_zt_reg<double, LZ, LT, B>;                                       \
    r.columns = B;                                                                  \
    r.threads = zt_reg_threads<double, LZ, LT, B>();                                \
    r.smem = zt_reg_smem<double, LZ, LT, B>();                                      \
  }
#define GFIX_Q(LZ, LT, B, W)                                                        \
  if (lz == LZ && lt == LT && lx % B == 0 && (want ? want == B : !r.fn)) {          \
    r.fn = k_fft_zt_quad<double, LZ, LT, B, W>;                                     \
    r.columns = B;                                                                  \
    r.threads = 4 * LZ * W;                                                         \
    r.smem = zt_reg_smem<double, LZ, LT, W>();                                      \
  }
  GFIX_Q(32, 64, 4, 2) GFIX_Q(36, 72, 2, 2) GFIX_Q(40, 80, 2, 2) GFIX_Q(48, 96, 2, 2)
  GFIX_T(4, 4, 4) GFIX_T(4, 8, 4) GFIX_T(8, 8, 4) GFIX_T(8, 16, 4) GFIX_T(12, 12, 4)
  GFIX_T(12, 24, 4) GFIX_T(16, 16, 4) GFIX_T(16, 32, 4) GFIX_T(20, 20, 4) GFIX_T(20, 40, 4)
  GFIX_T(24, 24, 4) GFIX_T(24, 48, 4) GFIX_T(4, 4, 2) GFIX_T(4, 8, 2) GFIX_T(8, 8, 2)
  GFIX_T(8, 16, 2) GFIX_T(16, 16, 2) GFIX_T(16, 32, 2) GFIX_T(24, 48, 2) GFIX_T(32, 32, 2)
  GFIX_T(28, 28, 4) GFIX_T(32, 32, 4)
  GFIX_T(6, 6, 2) GFIX_T(6, 12, 2) GFIX_T(10, 10, 2) GFIX_T(10, 20, 2) GFIX_T(14, 14, 2)
  GFIX_T(14, 28, 2) GFIX_T(18, 18, 2) GFIX_T(30, 30, 2)
  GFIX_T(18, 36, 2) GFIX_T(28, 56, 2) GFIX_T(30, 60, 2)
  GFIX_T(32, 64, 2) GFIX_T(32, 64, 1)
#undef GFIX_Q
#undef GFIX_T
  return r;
}

template <>
RegZt<double> reg_z<double>(int lz) {
  RegZt<double> r;
#define GFIX_Z(N)                    \
  if (lz == N) {                     \
    r.fn = k_fft_z_reg<double, N>;   \
    r.threads = kZThreads;           \
  }
  GFIX_Z(4) GFIX_Z(6) GFIX_Z(8) GFIX_Z(10) GFIX_Z(12) GFIX_Z(14) GFIX_Z(16) GFIX_Z(18)
  GFIX_Z(20) GFIX_Z(24)
#undef GFIX_Z
  return r;
}

}  // namespace gfix
