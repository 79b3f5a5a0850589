// fft_rows.h -- sizes shared by the two precisions' transform kernels (fft.cu, fft32.cu).
#pragma once

namespace pmpic {
namespace {

constexpr int FFT_THREADS = 256;  // Stockham kernels
constexpr int FS_THREADS = 128;   // four-step x passes

inline int pick_txf(int nx) {  // columns per CTA of the Stockham y passes
  if (nx % 16 == 0) return 16;
  if (nx % 8 == 0) return 8;
  if (nx % 4 == 0) return 4;
  return 2;
}
inline int pick_rp(int n) {  // complex rows per CTA of the Stockham x passes
  int rp = 4096 / n;
  if (rp < 1) rp = 1;
  if (rp > 8) rp = 8;
  return rp;
}

}  // namespace
}  // namespace pmpic
