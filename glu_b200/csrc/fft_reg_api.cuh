// The register-pencil passes (fft_reg.cuh) by extents.  They are compiled in
// translation units of their own, one for each pass and type (fft_xy_f32.cu
// .. fft_zt_f64.cu), for the extents listed there: 4 to 32, some up to
// 64, and t axes of once or twice the z extent.
#pragma once

#include "kernels.cuh"

namespace gfix {

// a pass: forward and inverse kernels (the same where it has one), the block
// and its shared memory; fn[0] null where there is none
template <typename R>
struct RegXy {
  void (*fn[2])(Ctx<R>, int, int) = {nullptr, nullptr};
  int planes = 1, threads = 0;  // planes of a block
  size_t smem = 0;
};
template <typename R>
struct RegZt {
  void (*fn)(Ctx<R>) = nullptr;
  int columns = 1, threads = 0;  // x columns of a block (Coulomb: any)
  size_t smem = 0;
};

// xy planes of n x n, in runs of `per` planes that a block may not cross
template <typename R>
RegXy<R> reg_xy(int n, int per);
// (z, t) tiles, of `want` columns or (0) the default width
template <typename R>
RegZt<R> reg_zt(int lz, int lt, int lx, int want);
// z of Coulomb slices
template <typename R>
RegZt<R> reg_z(int lz);

template <> RegXy<float> reg_xy<float>(int, int);
template <> RegXy<double> reg_xy<double>(int, int);
template <> RegZt<float> reg_zt<float>(int, int, int, int);
template <> RegZt<double> reg_zt<double>(int, int, int, int);
template <> RegZt<float> reg_z<float>(int);
template <> RegZt<double> reg_z<double>(int);

}  // namespace gfix
