// fft_impl.cuh -- the transform kernels of fft.cu, written once over the
// scalar type `real` (with `real2` its complex pair and mk2 its constructor)
// and included by fft.cu into one namespace per precision: FP64 for the plain
// path, FP32 for the mixed-precision form.  Not a standalone header.
__device__ __forceinline__ real2 cmul(real2 a, real2 b) {
  return mk2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ real2 cadd(real2 a, real2 b) { return mk2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ real2 csub(real2 a, real2 b) { return mk2(a.x - b.x, a.y - b.y); }

// forward DFT of size R in registers (exp(-2 pi i rt/R))
template <int R>
__device__ __forceinline__ void small_dft(real2* a) {
  if (R == 2) {
    real2 t0 = cadd(a[0], a[1]), t1 = csub(a[0], a[1]);
    a[0] = t0; a[1] = t1;
  } else if (R == 4) {
    real2 t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
    real2 t2 = cadd(a[1], a[3]), t3 = csub(a[1], a[3]);
    real2 mt3 = mk2(t3.y, -t3.x);  // -i * t3
    a[0] = cadd(t0, t2);
    a[2] = csub(t0, t2);
    a[1] = cadd(t1, mt3);
    a[3] = csub(t1, mt3);
  } else if (R == 3) {
    const real s3 = 0.86602540378443864676;  // sin(2pi/3)
    real2 s = cadd(a[1], a[2]), d = csub(a[1], a[2]);
    real2 b0 = cadd(a[0], s);
    real2 m = mk2(a[0].x - real(0.5) * s.x, a[0].y - real(0.5) * s.y);
    real2 r = mk2(s3 * d.y, -s3 * d.x);  // -i sin(2pi/3) d
    a[0] = b0;
    a[1] = cadd(m, r);
    a[2] = csub(m, r);
  } else if (R == 5) {
    const real c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
    const real s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
    real2 t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]);
    real2 t3 = csub(a[1], a[4]), t4 = csub(a[2], a[3]);
    real2 b0 = cadd(a[0], cadd(t1, t2));
    real2 m1 = mk2(a[0].x + c1 * t1.x + c2 * t2.x, a[0].y + c1 * t1.y + c2 * t2.y);
    real2 m2 = mk2(a[0].x + c2 * t1.x + c1 * t2.x, a[0].y + c2 * t1.y + c1 * t2.y);
    // -i (s1 t3 + s2 t4) and -i (s2 t3 - s1 t4)
    real2 n1 = mk2(s1 * t3.y + s2 * t4.y, -(s1 * t3.x + s2 * t4.x));
    real2 n2 = mk2(s2 * t3.y - s1 * t4.y, -(s2 * t3.x - s1 * t4.x));
    a[0] = b0;
    a[1] = cadd(m1, n1);
    a[4] = csub(m1, n1);
    a[2] = cadd(m2, n2);
    a[3] = csub(m2, n2);
  }
}

template <int R>
__device__ __forceinline__ void stage(const real2* __restrict__ src, real2* __restrict__ dst, int n, int len,
                                      int nrows, int stride_row, const real2* __restrict__ tw) {
  const int m = len / R, s = n / len;
  const int nb = m * s;  // butterflies per row
  for (int e = threadIdx.x; e < nb * nrows; e += blockDim.x) {
    int row = e / nb, b = e - row * nb;
    int p = b / s, q = b - p * s;
    const real2* S = src + (size_t)row * stride_row;
    real2* D = dst + (size_t)row * stride_row;
    real2 a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = S[q + s * (p + r * m)];
    small_dft<R>(a);
    D[q + s * (R * p)] = a[0];
#pragma unroll
    for (int t = 1; t < R; ++t) D[q + s * (R * p + t)] = cmul(a[t], tw[p * R + t]);
  }
}

// Forward complex FFT of nrows rows held in buf0 (stride_row); buf1 is the
// ping-pong workspace.  Returns the buffer holding the result.
__device__ real2* fft_rows(real2* buf0, real2* buf1, int nrows, int stride_row, const FftPlan& pl,
                             const real2* __restrict__ twbase) {
  real2* src = buf0;
  real2* dst = buf1;
  int len = pl.n;
  for (int st = 0; st < pl.nst; ++st) {
    const real2* tw = twbase + pl.tw_off[st];
    switch (pl.radix[st]) {
      case 4: stage<4>(src, dst, pl.n, len, nrows, stride_row, tw); break;
      case 2: stage<2>(src, dst, pl.n, len, nrows, stride_row, tw); break;
      case 3: stage<3>(src, dst, pl.n, len, nrows, stride_row, tw); break;
      case 5: stage<5>(src, dst, pl.n, len, nrows, stride_row, tw); break;
    }
    __syncthreads();
    len /= pl.radix[st];
    real2* t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// ---- forward y pass: phys -> mid ------------------------------------------------
// CTA: one z level, TXF consecutive x columns (TXF/2 complex rows of length Ny).
__global__ void __launch_bounds__(FFT_THREADS) k_fwd_y(Geom g, int TXF, FftPlan pl, const real2* __restrict__ tw,
                                                       const real* __restrict__ phys, real* __restrict__ mid) {
  PDL_WAIT();
  extern __shared__ real2 sm[];
  const int Ny = g.Ny, Nx = g.Nx;
  const int nr = TXF / 2;
  real2* b0 = sm;
  real2* b1 = sm + (size_t)nr * Ny;
  const int x0 = blockIdx.x * TXF, k = blockIdx.y;
  const real* P = phys + (size_t)k * Ny * Nx;
  for (int e = threadIdx.x; e < Ny * TXF; e += blockDim.x) {
    int j = e / TXF, x = e - j * TXF;
    real v = P[(size_t)j * Nx + x0 + x];
    real* c = (real*)&b0[(x >> 1) * Ny + j];
    c[x & 1] = v;
  }
  __syncthreads();
  real2* res = fft_rows(b0, b1, nr, Ny, pl, tw);
  real* M = mid + (size_t)k * g.sy * Nx;
  const int half = Ny / 2 + 1;
  for (int e = threadIdx.x; e < half * TXF; e += blockDim.x) {
    int a = e / TXF, x = e - a * TXF;
    int r = x >> 1;
    real2 z1 = res[r * Ny + a];
    real2 z2 = res[r * Ny + (a == 0 ? 0 : Ny - a)];
    real re, im;
    if ((x & 1) == 0) {  // A = (Z_a + conj Z_{N-a}) / 2
      re = real(0.5) * (z1.x + z2.x);
      im = real(0.5) * (z1.y - z2.y);
    } else {             // B = (Z_a - conj Z_{N-a}) / (2i)
      re = real(0.5) * (z1.y + z2.y);
      im = real(-0.5) * (z1.x - z2.x);
    }
    M[(size_t)(2 * a) * Nx + x0 + x] = re;
    M[(size_t)(2 * a + 1) * Nx + x0 + x] = im;
  }
}

// ---- forward x pass: mid -> spec ------------------------------------------------
// CTA: RP pairs of consecutive rows (row = (k, j') flattened), rows of length Nx.
__global__ void __launch_bounds__(FFT_THREADS) k_fwd_x(Geom g, int RP, int64_t nrows_total, FftPlan pl,
                                                       const real2* __restrict__ tw, const real* __restrict__ mid,
                                                       real* __restrict__ spec) {
  PDL_WAIT();
  extern __shared__ real2 sm[];
  const int Nx = g.Nx;
  real2* b0 = sm;
  real2* b1 = sm + (size_t)RP * Nx;
  const int64_t row0 = (int64_t)blockIdx.x * RP * 2;
  for (int e = threadIdx.x; e < RP * 2 * Nx; e += blockDim.x) {
    int rr = e / Nx, i = e - rr * Nx;
    int64_t row = row0 + rr;
    real v = row < nrows_total ? mid[(size_t)row * Nx + i] : real(0);
    real* c = (real*)&b0[(rr >> 1) * Nx + i];
    c[rr & 1] = v;
  }
  __syncthreads();
  real2* res = fft_rows(b0, b1, RP, Nx, pl, tw);
  const int half = Nx / 2 + 1;
  for (int e = threadIdx.x; e < RP * 2 * half; e += blockDim.x) {
    int rr = e / half, b = e - rr * half;
    int64_t row = row0 + rr;
    if (row >= nrows_total) continue;
    int r = rr >> 1;
    real2 z1 = res[r * Nx + b];
    real2 z2 = res[r * Nx + (b == 0 ? 0 : Nx - b)];
    real re, im;
    if ((rr & 1) == 0) {
      re = real(0.5) * (z1.x + z2.x);
      im = real(0.5) * (z1.y - z2.y);
    } else {
      re = real(0.5) * (z1.y + z2.y);
      im = real(-0.5) * (z1.x - z2.x);
    }
    spec[(size_t)row * g.sx + 2 * b] = re;
    spec[(size_t)row * g.sx + 2 * b + 1] = im;
  }
}

// Build Z_k = A_k + i B_k over the full circle from two half spectra, applying
// ffte_c2r's conjugate-symmetric fill (ffte_mod.F90:108-113): for k > N/2,
// A_k = conj(A_{N-k}); the imaginary parts of modes 0 and N/2 never reach the
// real output, so they are dropped.  Stored conjugated (FFTE computes the
// inverse as conj(FFT(conj(Z)))/N, vzfft1d.f:41-46, 63-68).
__device__ __forceinline__ real2 c2r_pack(real2 A, real2 B, int k, int n) {
  // A, B are the half-spectrum values at min(k, n-k); mirrored if k > n/2
  if (k == 0 || 2 * k == n) {
    A.y = real(0);
    B.y = real(0);
  }
  real2 z;
  if (2 * k <= n) {
    z = mk2(A.x - B.y, A.y + B.x);  // A + iB
  } else {
    // conj(A) + i conj(B) = (A.x + B.y) + i(-A.y + B.x)
    z = mk2(A.x + B.y, -A.y + B.x);
  }
  return mk2(z.x, -z.y);  // conj for the forward-transform inverse
}

// The spectral values A (row ra) and B (row ra + 1) of x mode km as the
// inverse x pass reads them, with the input operator applied.  ra is even and
// Ny + 2 is even, so row ra holds the even y' index jp (the real part of a y
// mode) and row ra + 1 the odd one of the same level lev; each value is the
// element pair (2 km, 2 km + 1) of its row.  The operators repeat the
// arithmetic of diffx and diffy (spectral.cu: dx_of, dy_of).
__device__ __forceinline__ real2 ld2(const real* __restrict__ p, size_t i) { return *(const real2*)&p[i]; }
__device__ __forceinline__ void st2(real* __restrict__ p, size_t i, real2 v) { *(real2*)&p[i] = v; }

// one array of a batch (selected without indexing the parameter arrays: no local copy)
template <class T>
__device__ __forceinline__ T* pick(T* const (&p)[6], int b) {
  return b < 3 ? (b == 0 ? p[0] : (b == 1 ? p[1] : p[2])) : (b == 3 ? p[3] : (b == 4 ? p[4] : p[5]));
}

// The operator on the values of one spectral element pair of rows ra (xa) and
// ra + 1 (xb); ca, cb are their spectral columns, x2 = 2 km the pair's x
// index.  The wavenumber tables are laid out like the spectra but kx depends
// on the x index alone and ky on the row alone, so kx is read from row 0 and
// ky from column 0 of rows ca - x2 and cb - x2: the same values, one small
// L1-resident row or a per-thread constant instead of a second spectrum-sized
// read per element.
template <int OP>
__device__ __forceinline__ void spec_op(const SpecIn<real>& S, real2 xa, real2 xb, int ca, int cb, int x2, real2& A,
                                        real2& B) {
  if constexpr (OP == SPEC_DX) {
    const real2 t = ld2(S.kx, x2);
    A = mk2((real(-1) * xa.y) * t.x, xa.x * t.y);
    B = mk2((real(-1) * xb.y) * t.x, xb.x * t.y);
  } else if constexpr (OP == SPEC_DY) {
    const real ta = S.ky[ca - x2], tb = S.ky[cb - x2];
    A = mk2((real(-1) * xb.x) * ta, (real(-1) * xb.y) * ta);
    B = mk2(xa.x * tb, xa.y * tb);
  } else {
    A = xa;
    B = xb;
  }
}

// the output operator of an inverse transform at physical element i, v the
// transformed value: the pointwise updates of vorticity_tendency.F90 in its
// order of operations (dp :169-171, :180-181, :191-193; dq :213-214,
// :224-225, :235-237; dr :250-264, with v = dw/dy)
template <int OP>
__device__ __forceinline__ real phys_op(const PhysOut<real>& E, size_t i, real v, real& o2) {
  const real o = E.o[i];
  if constexpr (OP == PHYS_ADD_MUL) return o + E.in[0][i] * v;
  if constexpr (OP == PHYS_ADD_MUL_SUM) return o + E.in[0][i] * (E.in[1][i] + v);
  if constexpr (OP == PHYS_NEG_ADD_MUL) return -o + E.in[0][i] * v;
  if constexpr (OP == PHYS_DQ_DR) {
    const real r = E.in[0][i], p = E.in[1][i];
    real w = p * E.in[3][i];
    w = w + E.in[2][i] * v;
    w = w + r * (-E.in[4][i]);
    w = w + r * (-E.in[5][i]);
    o2 = w;
    return o + r * (-p + v);
  }
  return o;
}
// one element, the operator chosen at run time (generic-length path)
__device__ __forceinline__ void phys_out_rt(const PhysOut<real>& E, real* __restrict__ phys, size_t i, real v) {
  if (E.op == PHYS_STORE || E.store) phys[i] = v;
  real w = real(0);
  switch (E.op) {
    case PHYS_ADD_MUL: E.o[i] = phys_op<PHYS_ADD_MUL>(E, i, v, w); break;
    case PHYS_ADD_MUL_SUM: E.o[i] = phys_op<PHYS_ADD_MUL_SUM>(E, i, v, w); break;
    case PHYS_NEG_ADD_MUL: E.o[i] = phys_op<PHYS_NEG_ADD_MUL>(E, i, v, w); break;
    case PHYS_DQ_DR:
      E.o[i] = phys_op<PHYS_DQ_DR>(E, i, v, w);
      E.o2[i] = w;
      break;
    default: break;
  }
}

// ---- inverse x pass: spec -> mid ------------------------------------------------
// (one array, batch entry q)
template <int OP>
__global__ void __launch_bounds__(FFT_THREADS) k_inv_x(Geom g, int RP, int64_t nrows_total, FftPlan pl,
                                                       const real2* __restrict__ tw, real* __restrict__ mid,
                                                       SpecIn<real> S, int q) {
  PDL_WAIT();
  extern __shared__ real2 sm[];
  const int Nx = g.Nx;
  real2* b0 = sm;
  real2* b1 = sm + (size_t)RP * Nx;
  const int64_t row0 = (int64_t)blockIdx.x * RP * 2;
  for (int e = threadIdx.x; e < RP * Nx; e += blockDim.x) {
    int r = e / Nx, k = e - r * Nx;
    int km = (2 * k <= Nx) ? k : Nx - k;
    int64_t ra = row0 + 2 * r;
    real2 A = mk2(real(0), real(0)), B = mk2(real(0), real(0));
    if (ra < nrows_total) {
      const int jp = (int)(ra % g.sy), ca = jp * g.sx + 2 * km;
      const size_t ea = (size_t)ra * g.sx + 2 * km;
      const real* x = pick(S.x, q);
      spec_op<OP>(S, ld2(x, ea), ld2(x, ea + g.sx), ca, ca + g.sx, 2 * km, A, B);
    }
    b0[r * Nx + k] = c2r_pack(A, B, k, Nx);
  }
  __syncthreads();
  real2* res = fft_rows(b0, b1, RP, Nx, pl, tw);
  const real dn = real(1) / (real)Nx;
  for (int e = threadIdx.x; e < RP * 2 * Nx; e += blockDim.x) {
    int rr = e / Nx, i = e - rr * Nx;
    int64_t row = row0 + rr;
    if (row >= nrows_total) continue;
    real2 z = res[(rr >> 1) * Nx + i];
    // conj(z) * dn: real part -> row A, imaginary part -> row B
    mid[(size_t)row * Nx + i] = (rr & 1) == 0 ? z.x * dn : -z.y * dn;
  }
}

// ---- inverse y pass: mid -> phys ------------------------------------------------
__global__ void __launch_bounds__(FFT_THREADS) k_inv_y(Geom g, int TXF, FftPlan pl,
                                                       const real2* __restrict__ tw, const real* __restrict__ mid,
                                                       real* __restrict__ phys, PhysOut<real> E) {
  PDL_WAIT();
  extern __shared__ real2 sm[];
  const int Ny = g.Ny, Nx = g.Nx;
  const int nr = TXF / 2;
  real2* b0 = sm;
  real2* b1 = sm + (size_t)nr * Ny;
  const int x0 = blockIdx.x * TXF, k = blockIdx.y;
  const real* M = mid + (size_t)k * g.sy * Nx;
  // stage the half spectra (Ny/2+1 modes x TXF columns) into b1 first
  const int half = Ny / 2 + 1;
  for (int e = threadIdx.x; e < half * TXF; e += blockDim.x) {
    int a = e / TXF, x = e - a * TXF;
    b1[x * half + a] = mk2(M[(size_t)(2 * a) * Nx + x0 + x], M[(size_t)(2 * a + 1) * Nx + x0 + x]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nr * Ny; e += blockDim.x) {
    int r = e / Ny, kk = e - r * Ny;
    int km = (2 * kk <= Ny) ? kk : Ny - kk;
    real2 A = b1[(2 * r) * half + km], B = b1[(2 * r + 1) * half + km];
    b0[r * Ny + kk] = c2r_pack(A, B, kk, Ny);
  }
  __syncthreads();
  real2* res = fft_rows(b0, b1, nr, Ny, pl, tw);
  const real dn = real(1) / (real)Ny;
  const size_t p0 = (size_t)k * Ny * Nx;
  for (int e = threadIdx.x; e < Ny * TXF; e += blockDim.x) {
    int j = e / TXF, x = e - j * TXF;
    real2 z = res[(x >> 1) * Ny + j];
    phys_out_rt(E, phys, p0 + (size_t)j * Nx + x0 + x, (x & 1) == 0 ? z.x * dn : -z.y * dn);
  }
}

// ---- four-step register FFT for n = n1 * n2, n1 and n2 in 2 .. 16 ---------------------
// x[n2 + N2 n1] -> X[k1 + N1 k2]:  n1-point DFTs over n1 (one thread per n2),
// twiddle W_n^(n2 k1), transpose through shared memory, n2-point DFTs over n2
// (one thread per k1).  The small DFTs run in registers; loads and stores touch
// global memory once each.
// The kernels are instantiated for the splits (N1c, N2c) of FS_SPLITS and once
// for every other length with the split read at run time (N1c = N2c = 0): the
// radix then selects among the register DFTs by a branch that is uniform over
// the grid.  What bounds them, by counters at 128^3: the FP32 x passes L1
// (62-74% of its throughput), the FP64 ones L1 (46-59%) and the latency of few
// warps (17-29% active); the y passes the latency of a row's loads and
// barriers (33-47% of L1, 17-36% of DRAM).  The twiddles are laid out [k1][n2],
// so that the lanes of a warp, which differ in n2, read one line.

// W_16^m = exp(-2 pi i m / 16), m known at compile time after unrolling
__device__ __forceinline__ real2 w16(int m) {
  constexpr real C1 = 0.92387953251128675613;  // cos(pi/8)
  constexpr real C2 = 0.70710678118654752440;  // cos(pi/4)
  constexpr real C3 = 0.38268343236508977173;  // cos(3pi/8)
  switch (m & 15) {
    case 0: return mk2(1.0, 0.0);
    case 1: return mk2(C1, -C3);
    case 2: return mk2(C2, -C2);
    case 3: return mk2(C3, -C1);
    case 4: return mk2(0.0, -1.0);
    case 5: return mk2(-C3, -C1);
    case 6: return mk2(-C2, -C2);
    case 7: return mk2(-C1, -C3);
    case 8: return mk2(-1.0, 0.0);
    case 9: return mk2(-C1, C3);
    case 10: return mk2(-C2, C2);
    case 11: return mk2(-C3, C1);
    case 12: return mk2(0.0, 1.0);
    case 13: return mk2(C3, C1);
    case 14: return mk2(C2, C2);
    default: return mk2(C1, C3);
  }
}
// W_R^m for the other composite radices, R = 6, 9, 10, 12, 15 (m <= 8 occurs)
template <int R>
__device__ __forceinline__ real2 wr(int m) {
  if constexpr (R == 6) {
    switch (m) {
      case 1: return mk2(0.5, -0.866025403784438646764);
      default: return mk2(-0.5, -0.866025403784438646764);
    }
  } else if constexpr (R == 9) {
    switch (m) {
      case 1: return mk2(0.766044443118978035202, -0.642787609686539326323);
      case 2: return mk2(0.173648177666930348852, -0.984807753012208059367);
      case 3: return mk2(-0.5, -0.866025403784438646764);
      default: return mk2(-0.939692620785908384054, -0.342020143325668733044);
    }
  } else if constexpr (R == 10) {
    switch (m) {
      case 1: return mk2(0.809016994374947424102, -0.587785252292473129169);
      case 2: return mk2(0.309016994374947424102, -0.951056516295153572116);
      case 3: return mk2(-0.309016994374947424102, -0.951056516295153572116);
      default: return mk2(-0.809016994374947424102, -0.587785252292473129169);
    }
  } else if constexpr (R == 12) {
    switch (m) {
      case 1: return mk2(0.866025403784438646764, -0.5);
      case 2: return mk2(0.5, -0.866025403784438646764);
      case 3: return mk2(0.0, -1.0);
      case 4: return mk2(-0.5, -0.866025403784438646764);
      case 5: return mk2(-0.866025403784438646764, -0.5);
      default: return mk2(-1.0, 0.0);
    }
  } else {
    switch (m) {
      case 1: return mk2(0.913545457642600895502, -0.406736643075800207754);
      case 2: return mk2(0.669130606358858213826, -0.743144825477394235015);
      case 3: return mk2(0.309016994374947424102, -0.951056516295153572116);
      case 4: return mk2(-0.104528463267653471400, -0.994521895368273336923);
      case 5: return mk2(-0.5, -0.866025403784438646764);
      case 6: return mk2(-0.809016994374947424102, -0.587785252292473129169);
      case 7: return mk2(-0.978147600733805637929, -0.207911690817759337102);
      default: return mk2(-0.978147600733805637929, 0.207911690817759337102);
    }
  }
}

// the first of the (one or two) stages of a register radix, in the Stockham
// path's order 4, 2, 3, 5
__host__ __device__ constexpr int first_stage(int R) {
  return R <= 5 ? R : (R % 4 == 0 ? 4 : (R % 2 == 0 ? 2 : 3));
}
// forward DFT of size R in registers, natural order in and out: composite
// sizes as M1 x M2 with the constants above (8 = 4 x 2, 16 = 4 x 4, 6 = 2 x 3,
// 9 = 3 x 3, 10 = 2 x 5, 12 = 4 x 3, 15 = 3 x 5)
template <int R>
__device__ __forceinline__ void dft(real2* a) {
  if constexpr (R <= 5) {
    small_dft<R>(a);
  } else {
    constexpr int M1 = first_stage(R), M2 = R / M1;
    real2 y[R];
#pragma unroll
    for (int n2 = 0; n2 < M2; ++n2) {
      real2 b[M1];
#pragma unroll
      for (int n1 = 0; n1 < M1; ++n1) b[n1] = a[M2 * n1 + n2];
      small_dft<M1>(b);
#pragma unroll
      for (int k1 = 0; k1 < M1; ++k1) {
        if (n2 * k1 == 0) y[k1 * M2 + n2] = b[k1];
        else if constexpr (R == 8 || R == 16) y[k1 * M2 + n2] = cmul(b[k1], w16(n2 * k1 * (16 / R)));
        else y[k1 * M2 + n2] = cmul(b[k1], wr<R>(n2 * k1));
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < M1; ++k1) {
      real2 c[M2];
#pragma unroll
      for (int n2 = 0; n2 < M2; ++n2) c[n2] = y[k1 * M2 + n2];
      small_dft<M2>(c);
#pragma unroll
      for (int k2 = 0; k2 < M2; ++k2) a[k1 + M1 * k2] = c[k2];
    }
  }
}
template <int R>
struct Rad {
  static constexpr int value = R;
};
// f(Rad<r>) for the radix r: known at compile time (RC > 0), or one of the radices of fs_split
template <int RC, class F>
__device__ __forceinline__ void with_radix(int r, F&& f) {
  if constexpr (RC > 0) {
    f(Rad<RC>{});
  } else {
    switch (r) {
      case 2: f(Rad<2>{}); break;
      case 3: f(Rad<3>{}); break;
      case 4: f(Rad<4>{}); break;
      case 5: f(Rad<5>{}); break;
      case 6: f(Rad<6>{}); break;
      case 8: f(Rad<8>{}); break;
      case 9: f(Rad<9>{}); break;
      case 10: f(Rad<10>{}); break;
      case 12: f(Rad<12>{}); break;
      case 15: f(Rad<15>{}); break;
      default: f(Rad<16>{}); break;
    }
  }
}
// step 1 of one row: a[n1] = x[n2 + N2 n1] on entry; Y row [k1][n2] (padded).
// ST: the first one or two stages of the Stockham path themselves, with its
// twiddles (the length's other stages are the step-3 DFTs): the radices and
// the order of the Stockham kernels.  Rows of the two differ at most where a
// composite DFT has a quarter turn exactly, (0, -1), and the table its rounding
// in long double, (-2.5e-20, -1): bits change only where the components of a
// value differ by a factor above 1000 (FP64).
// Otherwise an R-point DFT and the twiddle W_n^(n2 k1).
template <int R, bool ST>
__device__ __forceinline__ void fs_step1(real2* a, int n2, int N2, real2* Yrow, const real2* __restrict__ tw4) {
  if constexpr (ST) {
    constexpr int M1 = first_stage(R), M2 = R / M1;
    real2 y[R];
#pragma unroll
    for (int m = 0; m < M2; ++m) {
      real2 b[M1];
#pragma unroll
      for (int u = 0; u < M1; ++u) b[u] = a[M2 * u + m];
      small_dft<M1>(b);
#pragma unroll
      for (int k = 0; k < M1; ++k) y[k * M2 + m] = k == 0 ? b[k] : cmul(b[k], tw4[(m * M1 + k) * N2 + n2]);
    }
    const real2* __restrict__ t2 = tw4 + R * N2;
#pragma unroll
    for (int k1 = 0; k1 < M1; ++k1) {
      real2 c[M2];
#pragma unroll
      for (int m = 0; m < M2; ++m) c[m] = y[k1 * M2 + m];
      if constexpr (M2 > 1) small_dft<M2>(c);
#pragma unroll
      for (int k2 = 0; k2 < M2; ++k2)
        Yrow[(k1 + M1 * k2) * (N2 + 1) + n2] = k2 == 0 ? c[k2] : cmul(c[k2], t2[k2 * N2 + n2]);
    }
  } else {
    dft<R>(a);
#pragma unroll
    for (int k1 = 0; k1 < R; ++k1)
      Yrow[k1 * (N2 + 1) + n2] = (k1 == 0 || n2 == 0) ? a[k1] : cmul(a[k1], tw4[k1 * N2 + n2]);
  }
}
// step 3 of one row: a[k2] = X[k1 + N1 k2] on return
template <int R>
__device__ __forceinline__ void fs_step3(real2* a, int k1, const real2* Yrow) {
#pragma unroll
  for (int n2 = 0; n2 < R; ++n2) a[n2] = Yrow[k1 * (R + 1) + n2];
  dft<R>(a);
}
__host__ __device__ constexpr int FS_AM(int n1, int n2) { return n1 == 0 ? 16 : (n1 > n2 ? n1 : n2); }
// complex rows of an x pass's CTA, and the shared values of a CTA's rows: x
// passes pad rows to N1 (N2 + 1), y passes by one more, so
// that the column pairs of a warp fall in distinct banks
constexpr int FS_YV = 128 / sizeof(real2);  // a row's column pairs are one 128-byte line
constexpr int FS_YT = 16 * FS_YV;           // threads of a y pass's CTA at most
__host__ __device__ constexpr int fs_rows(int n1, int n2) { return FS_THREADS / (n1 > n2 ? n1 : n2); }
__host__ __device__ constexpr int fs_xvals(int n1, int n2) { return n1 == 0 ? 8 * 16 * 17 : fs_rows(n1, n2) * n1 * (n2 + 1); }
__host__ __device__ constexpr int fs_yvals(int n1, int n2) { return n1 == 0 ? FS_YV * (16 * 17 + 1) : FS_YV * (n1 * (n2 + 1) + 1); }

template <class T>
struct Arr6 {
  T* p[6];
};

// forward x pass (mid -> spec): pairs of real rows; blockIdx.y is the array of the batch
template <int N1c, int N2c, bool ST>
__global__ void __launch_bounds__(FS_THREADS) k4_fwd_x(Geom g, int n1, int n2_, int64_t nrows,
                                                       const real2* __restrict__ tw4, Arr6<const real> mids,
                                                       Arr6<real> specs) {
  PDL_WAIT();
  const int N1 = N1c ? N1c : n1, N2 = N2c ? N2c : n2_, N = N1 * N2;
  const int RP = FS_THREADS / (N1 > N2 ? N1 : N2), YS = N1 * (N2 + 1);
  __shared__ real2 Y[fs_xvals(N1c, N2c)];
  real2* X = Y;  // [RP][N], reuses Y after step 3 has read it
  const real* __restrict__ mid = pick(mids.p, blockIdx.y);
  real* __restrict__ spec = pick(specs.p, blockIdx.y);
  const int t = threadIdx.x;
  const int64_t row0 = (int64_t)blockIdx.x * RP * 2;
  real2 a[FS_AM(N1c, N2c)];
  if (t < RP * N2) {
    const int r = t / N2, n2 = t - r * N2;
    const int64_t ra = row0 + 2 * r, rb = ra + 1;
    with_radix<N1c>(N1, [&](auto rad) {
      constexpr int R = decltype(rad)::value;
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int i = n2 + N2 * u;
        a[u] = mk2(ra < nrows ? mid[(size_t)ra * N + i] : real(0), rb < nrows ? mid[(size_t)rb * N + i] : real(0));
      }
      fs_step1<R, ST>(a, n2, N2, Y + r * YS, tw4);
    });
  }
  __syncthreads();
  const bool act = t < RP * N1;  // every thread reaches the barriers
  const int r = t / N1, k1 = t - r * N1;
  if (act) with_radix<N2c>(N2, [&](auto rad) { fs_step3<decltype(rad)::value>(a, k1, Y + r * YS); });
  __syncthreads();
  if (act)
    with_radix<N2c>(N2, [&](auto rad) {
#pragma unroll
      for (int k2 = 0; k2 < decltype(rad)::value; ++k2) X[r * N + k1 + N1 * k2] = a[k2];
    });
  __syncthreads();
  // separate the two real rows: A = (Z_b + conj Z_{N-b}) / 2, B = (Z_b - conj Z_{N-b}) / (2i)
  const int HALF = N / 2 + 1;
  for (int e = t; e < RP * 2 * HALF; e += FS_THREADS) {
    const int rr = e / HALF, b = e - rr * HALF;
    const int64_t row = row0 + rr;
    if (row >= nrows) continue;
    const int rz = rr >> 1;
    const real2 z1 = X[rz * N + b];
    const real2 z2 = X[rz * N + (b == 0 ? 0 : N - b)];
    real2 v;
    if ((rr & 1) == 0) v = mk2(real(0.5) * (z1.x + z2.x), real(0.5) * (z1.y - z2.y));
    else v = mk2(real(0.5) * (z1.y + z2.y), real(-0.5) * (z1.x - z2.x));
    st2(spec, (size_t)row * g.sx + 2 * b, v);
  }
}

// Inverse x pass (spec -> mid).  The modes are read straight from HBM into
// registers (the mirrored half from L1), the input operator applied on the
// way.  SPEC_PAIR transforms the x and the y derivative of a spectrum from one
// read of it.
template <int N1c, int N2c, bool ST, int OP>
__global__ void __launch_bounds__(FS_THREADS, sizeof(real) == 4 ? 5 : 3) k4_inv_x(Geom g, int n1, int n2_, int64_t nrows,
                                                       const real2* __restrict__ tw4, SpecIn<real> S,
                                                       Arr6<real> mids, Arr6<real> ymids) {
  PDL_WAIT();
  const int N1 = N1c ? N1c : n1, N2 = N2c ? N2c : n2_, N = N1 * N2;
  const int RP = FS_THREADS / (N1 > N2 ? N1 : N2), YS = N1 * (N2 + 1);
  extern __shared__ real2 sm[];
  real2* Y = sm;
  real2* Yd = sm + RP * YS;  // SPEC_PAIR: the y derivative
  const int q = blockIdx.y;
  const int t = threadIdx.x;
  const int64_t row0 = (int64_t)blockIdx.x * RP * 2;
  real2 a[FS_AM(N1c, N2c)];
  if (t < RP * N2) {
    const int r = t / N2, n2 = t - r * N2;
    const int64_t ra = row0 + 2 * r;
    const bool valid = ra < nrows;  // then so is ra + 1: the row count is even
    const int jp = (int)(ra % g.sy);
    const real* __restrict__ x = pick(S.x, q);
    with_radix<N1c>(N1, [&](auto rad) {
      constexpr int R = decltype(rad)::value;
      [[maybe_unused]] real2 b[OP == SPEC_PAIR ? R : 1];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int k = n2 + N2 * u;
        const int km = (2 * k <= N) ? k : N - k;
        const int ca = jp * g.sx + 2 * km, cb = ca + g.sx;
        real2 xa = mk2(real(0), real(0)), xb = xa, A, B;
        if (valid) {
          const size_t ea = (size_t)ra * g.sx + 2 * km;
          xa = ld2(x, ea);
          xb = ld2(x, ea + g.sx);
        }
        if constexpr (OP == SPEC_PAIR) {
          spec_op<SPEC_DY>(S, xa, xb, ca, cb, 2 * km, A, B);
          b[u] = c2r_pack(A, B, k, N);
          spec_op<SPEC_DX>(S, xa, xb, ca, cb, 2 * km, A, B);
        } else {
          spec_op<OP>(S, xa, xb, ca, cb, 2 * km, A, B);
        }
        a[u] = c2r_pack(A, B, k, N);
      }
      fs_step1<R, ST>(a, n2, N2, Y + r * YS, tw4);
      if constexpr (OP == SPEC_PAIR) fs_step1<R, ST>(b, n2, N2, Yd + r * YS, tw4);
    });
  }
  __syncthreads();
  const real dn = real(1) / (real)N;
  if (t < RP * N1) {
    const int r = t / N1, k1 = t - r * N1;
    const int64_t ra = row0 + 2 * r, rb = ra + 1;
    with_radix<N2c>(N2, [&](auto rad) {
      constexpr int R = decltype(rad)::value;
      auto out = [&](const real2* src, real* __restrict__ mid) {
        fs_step3<R>(a, k1, src + r * YS);
#pragma unroll
        for (int k2 = 0; k2 < R; ++k2) {
          const int i = k1 + N1 * k2;  // conj(z) * dn: real part -> row A, imaginary part -> row B
          if (ra < nrows) mid[(size_t)ra * N + i] = a[k2].x * dn;
          if (rb < nrows) mid[(size_t)rb * N + i] = -a[k2].y * dn;
        }
      };
      out(Y, pick(mids.p, q));
      if constexpr (OP == SPEC_PAIR) out(Yd, pick(ymids.p, q));
    });
  }
}

// forward y pass (phys -> mid): one z level, FS_YV consecutive pairs of x
// columns per CTA; thread order puts consecutive x on consecutive threads, so
// a warp's access is whole 128-byte lines (FP32 with 8 pairs, half lines: 4
// instead of 2 lines an access)
template <int N1c, int N2c, bool ST>
__global__ void __launch_bounds__(FS_YT) k4_fwd_y(Geom g, int n1, int n2_,
                                                       const real2* __restrict__ tw4, Arr6<const real> physs,
                                                       Arr6<real> mids) {
  PDL_WAIT();
  const int N1 = N1c ? N1c : n1, N2 = N2c ? N2c : n2_, N = N1 * N2;
  constexpr int RP = FS_YV;
  const int YS = N1 * (N2 + 1) + 1, XS = N + 1;
  __shared__ real2 Y[fs_yvals(N1c, N2c)];
  real2* X = Y;  // [RP][XS], reuses Y after step 3 has read it
  const int t = threadIdx.x, Nx = g.Nx;
  const int x0 = blockIdx.x * 2 * RP, k = blockIdx.y;
  const real* __restrict__ P = pick(physs.p, blockIdx.z) + (size_t)k * N * Nx;
  real2 a[FS_AM(N1c, N2c)];
  const int r = t % RP;
  if (t < RP * N2) {
    const int n2 = t / RP;
    const bool in = x0 + 2 * r < Nx;
    with_radix<N1c>(N1, [&](auto rad) {
      constexpr int R = decltype(rad)::value;
#pragma unroll
      for (int u = 0; u < R; ++u)  // columns x0+2r (re), x0+2r+1 (im)
        a[u] = in ? ld2(P, (size_t)(n2 + N2 * u) * Nx + x0 + 2 * r) : mk2(real(0), real(0));
      fs_step1<R, ST>(a, n2, N2, Y + r * YS, tw4);
    });
  }
  __syncthreads();
  const bool act = t < RP * N1;  // every thread reaches the barriers
  const int k1 = t / RP;
  if (act) with_radix<N2c>(N2, [&](auto rad) { fs_step3<decltype(rad)::value>(a, k1, Y + r * YS); });
  __syncthreads();
  if (act)
    with_radix<N2c>(N2, [&](auto rad) {
#pragma unroll
      for (int k2 = 0; k2 < decltype(rad)::value; ++k2) X[r * XS + k1 + N1 * k2] = a[k2];
    });
  __syncthreads();
  const int HALF = N / 2 + 1;
  real* __restrict__ M = pick(mids.p, blockIdx.z) + (size_t)k * g.sy * Nx;
  for (int e = t; e < HALF * 2 * RP; e += blockDim.x) {
    const int m = e / (2 * RP), x = e - m * (2 * RP);
    if (x0 + x >= Nx) continue;
    const int rz = x >> 1;
    const real2 z1 = X[rz * XS + m];
    const real2 z2 = X[rz * XS + (m == 0 ? 0 : N - m)];
    real re, im;
    if ((x & 1) == 0) {
      re = real(0.5) * (z1.x + z2.x);
      im = real(0.5) * (z1.y - z2.y);
    } else {
      re = real(0.5) * (z1.y + z2.y);
      im = real(-0.5) * (z1.x - z2.x);
    }
    M[(size_t)(2 * m) * Nx + x0 + x] = re;
    M[(size_t)(2 * m + 1) * Nx + x0 + x] = im;
  }
}

// step 1 of an inverse y pass: the modes of column pair r read from M (a level
// of a mid array) into Y
// (FEW: at most eight modes' loads in flight, for a caller with sums in registers)
template <int N1c, bool ST, bool FEW = false>
__device__ __forceinline__ void inv_y_step1(const Geom& g, int N1, int N2, int t, int x0, const real* __restrict__ M,
                                            const real2* __restrict__ tw4, real2* a, real2* Y, int YS) {
  const int N = N1 * N2, Nx = g.Nx;
  const int r = t % FS_YV, n2 = t / FS_YV;
  if (n2 >= N2) return;
  const bool in = x0 + 2 * r < Nx;
  with_radix<N1c>(N1, [&](auto rad) {
    constexpr int R = decltype(rad)::value;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      if (FEW && u % (sizeof(real) == 4 ? 8 : 4) == 0) asm volatile("" ::: "memory");
      const int kk = n2 + N2 * u;
      const int km = (2 * kk <= N) ? kk : N - kk;
      real2 re = mk2(real(0), real(0)), im = re;
      if (in) {
        const uint32_t o = (uint32_t)(2 * km * Nx + x0 + 2 * r);  // within the level
        re = ld2(M, o);                                           // (A.re, B.re)
        im = ld2(M, o + Nx);                                      // (A.im, B.im)
      }
      a[u] = c2r_pack(mk2(re.x, im.x), mk2(re.y, im.y), kk, N);
    }
    fs_step1<R, ST>(a, n2, N2, Y + r * YS, tw4);
  });
}

// inverse y pass (mid -> phys); blockIdx.z is the array of the batch
template <int N1c, int N2c, bool ST>
__global__ void __launch_bounds__(FS_YT) k4_inv_y(Geom g, int n1, int n2_,
                                                       const real2* __restrict__ tw4, Arr6<const real> mids,
                                                       Arr6<real> physs) {
  PDL_WAIT();
  const int N1 = N1c ? N1c : n1, N2 = N2c ? N2c : n2_, N = N1 * N2;
  constexpr int RP = FS_YV;
  const int YS = N1 * (N2 + 1) + 1;
  __shared__ real2 Y[fs_yvals(N1c, N2c)];
  const int t = threadIdx.x, Nx = g.Nx;
  const int x0 = blockIdx.x * 2 * RP, k = blockIdx.y;
  real2 a[FS_AM(N1c, N2c)];
  inv_y_step1<N1c, ST>(g, N1, N2, t, x0, pick(mids.p, blockIdx.z) + (size_t)k * g.sy * Nx, tw4, a, Y, YS);
  __syncthreads();
  const real dn = real(1) / (real)N;
  const int r = t % RP, k1 = t / RP;
  if (k1 < N1 && x0 + 2 * r < Nx) {
    real* __restrict__ phys = pick(physs.p, blockIdx.z);
    const size_t p0 = (size_t)k * N * Nx + x0 + 2 * r;
    with_radix<N2c>(N2, [&](auto rad) {
      constexpr int R = decltype(rad)::value;
      fs_step3<R>(a, k1, Y + r * YS);
#pragma unroll
      for (int k2 = 0; k2 < R; ++k2) st2(phys, p0 + (size_t)(k1 + N1 * k2) * Nx, mk2(a[k2].x * dn, -a[k2].y * dn));
    });
  }
}

// The inverse y passes of vorticity_tendency's eight derivatives with its
// pointwise products, in one kernel: a CTA transforms the eight fields of its
// columns one after the other and sums dp, then dq, in registers, so that no
// derivative is stored and dp and dq are written once
// (vorticity_tendency.F90:147-265, in its order of operations):
//   dp = db/dy + p du/dx + q du/dy + r (q + dw/dx)
//   dq = -db/dx + p dv/dx + q dv/dy + r (-p + dw/dy)
//   dr = p dw/dx + q dw/dy - r du/dx - r dv/dy
// dr's products come in another order than its sum: they wait in dr and two
// work grids, each element with the thread that owns it.  The FP64 path's sums
// would take half of the registers: they wait in dp and dq themselves.  The
// exchange buffer alternates between two halves: one barrier a field.
// Measured, ms per step of the whole tendency (its eight y passes as kernels
// of their own before): FP32 256^3 5.1 -> 4.4, 128^3 0.96 -> 0.81; FP64 128^3
// 1.58 -> 1.30 (sums in registers 1.47); 32^3 0.57 -> 0.20.
struct VtArgs {
  const real* m[8];  // x-transformed db/dy, du/dx, du/dy, dw/dx, db/dx, dv/dx, dv/dy, dw/dy
  const real *P, *Q, *R;
  real *DP, *DQ, *DR, *tmp, *tmp2;
};
template <int N1c, int N2c, bool ST>
__global__ void __launch_bounds__(FS_YT, sizeof(real) == 4 ? 2 : 4) k4_vt_y(Geom g, int n1, int n2_,
                                                      const real2* __restrict__ tw4, const __grid_constant__ VtArgs V) {
  PDL_WAIT();
  const int N1 = N1c ? N1c : n1, N2 = N2c ? N2c : n2_, N = N1 * N2;
  constexpr int RP = FS_YV;
  constexpr bool MEM = sizeof(real) == 8;  // the sums wait in memory
  const int YS = N1 * (N2 + 1) + 1;
  extern __shared__ real2 sm[];
  const int t = threadIdx.x, Nx = g.Nx;
  const int x0 = blockIdx.x * 2 * RP, k = blockIdx.y;
  const int r = t % RP, k1 = t / RP;
  const bool act = k1 < N1 && x0 + 2 * r < Nx;
  const size_t lev = (size_t)k * N * Nx;
  const uint32_t p0 = (uint32_t)(k1 * Nx + x0 + 2 * r);  // within the level
  const real dn = real(1) / (real)N;
  real2 a[FS_AM(N1c, N2c)], acc[MEM ? 1 : FS_AM(N1c, N2c)];
#pragma unroll 1
  for (int f = 0; f < 8; ++f) {
    real2* Y = sm + (f & 1) * (RP * YS);
    inv_y_step1<N1c, ST, true>(g, N1, N2, t, x0, V.m[f] + (size_t)k * g.sy * Nx, tw4, a, Y, YS);
    __syncthreads();
    if (!act) continue;
    // field f adds X (Z + v) to the sum (Z: null, q or -p)
    const real* X = f == 1 || f == 5 ? V.P : (f == 2 || f == 6 ? V.Q : V.R);
    const real* Z = f == 3 ? V.Q : (f == 7 ? V.P : nullptr);
    const real sz = f == 7 ? real(-1) : real(1);
    real* sum = (f < 4 ? V.DP : V.DQ) + lev;
    with_radix<N2c>(N2, [&](auto rad) {
      constexpr int R = decltype(rad)::value;
      fs_step3<R>(a, k1, Y + r * YS);
#pragma unroll
      for (int k2 = 0; k2 < R; ++k2) {
        // (a few elements' loads in flight at a time: more would spill the sums)
        if (k2 % (sizeof(real) == 4 ? 4 : 2) == 0) asm volatile("" ::: "memory");
        const uint32_t o = p0 + (uint32_t)(N1 * k2 * Nx);
        const real2 v = mk2(a[k2].x * dn, -a[k2].y * dn);
        real2 s;
        if ((f & 3) == 0) {
          s = f == 0 ? v : mk2(-v.x, -v.y);
        } else {
          const real2 x = ld2(X + lev, o);
          real2 u = v;
          if (Z) {
            const real2 z = ld2(Z + lev, o);
            u = mk2(sz * z.x + v.x, sz * z.y + v.y);
          }
          s = MEM ? ld2(sum, o) : acc[MEM ? 0 : k2];
          s = mk2(s.x + x.x * u.x, s.y + x.y * u.y);
        }
        if (!MEM) acc[MEM ? 0 : k2] = s;
        if (MEM || (f & 3) == 3) st2(sum, o, s);
        if (f == 1) {
          const real2 w = ld2(V.R + lev, o);
          st2(V.DR + lev, o, mk2(w.x * -v.x, w.y * -v.y));
        } else if (f == 3) {
          const real2 w = ld2(V.P + lev, o);
          st2(V.tmp2 + lev, o, mk2(w.x * v.x, w.y * v.y));
        } else if (f == 6) {
          const real2 w = ld2(V.R + lev, o);
          st2(V.tmp + lev, o, mk2(w.x * -v.x, w.y * -v.y));
        } else if (f == 7) {
          const real2 w = ld2(V.Q + lev, o), d0 = ld2(V.tmp2 + lev, o), d1 = ld2(V.DR + lev, o), d2 = ld2(V.tmp + lev, o);
          st2(V.DR + lev, o, mk2(d0.x + w.x * v.x + d1.x + d2.x, d0.y + w.y * v.y + d1.y + d2.y));
        }
      }
    });
  }
}

// f(N1c, N2c, ST) for a plan: the lengths 2^k, 3 2^k, 5 2^k and 9 2^k of common
// grids at compile time, the others at run time (the same kernels, with the
// registers of the largest radix: both transforms of a step took 0.67 ms at
// 96^3 FP32 with the split known, 1.04 with it read at run time)
constexpr int FS_SPLITS[][3] = {{4, 4, 0},  {8, 4, 0},   {8, 8, 0}, {16, 8, 0}, {16, 16, 0}, {4, 6, 1}, {4, 12, 1},
                                {16, 6, 1}, {16, 12, 1}, {8, 5, 1}, {16, 5, 1}, {16, 10, 1}, {8, 9, 1}, {16, 9, 1}};
constexpr int FS_NSPLIT = sizeof(FS_SPLITS) / sizeof(FS_SPLITS[0]);
template <bool B>
struct Flag {
  static constexpr bool value = B;
};
template <int I = 0, class F>
void fs_dispatch(int n1, int n2, bool st, F&& f) {
  if constexpr (I == FS_NSPLIT) {
    f(Rad<0>{}, Rad<0>{}, Flag<true>{});
  } else {
    constexpr int A = FS_SPLITS[I][0], B = FS_SPLITS[I][1];
    constexpr bool S = FS_SPLITS[I][2] != 0;
    if (n1 == A && n2 == B && st == S) f(Rad<A>{}, Rad<B>{}, Flag<S>{});
    else fs_dispatch<I + 1>(n1, n2, st, f);
  }
}

// y then x pass of nb arrays (1..6); mids: nb scratch arrays
int fft_forward_impl(pmpic_ctx* ctx, int nb, const real* const* phys, real* const* spec, real* const* mids,
                     const real2* tw) {
  TimerScope ts(ctx, T_FFTF);
  const Geom& g = ctx->g;
  const FftPlan& px = ctx->plan_x;
  const FftPlan& py = ctx->plan_y;
  const real2* twy = tw + ctx->ftw_off_y;
  cudaStream_t st = ctx->stream;
  Arr6<const real> P{}, MC{};
  Arr6<real> M{}, Sp{};
  for (int b = 0; b < nb; ++b) {
    P.p[b] = phys[b];
    MC.p[b] = M.p[b] = mids[b];
    Sp.p[b] = spec[b];
  }
  const int64_t nrows = (int64_t)g.nzp * g.sy;
  if (py.n1) {
    const dim3 gr((g.Nx + 2 * FS_YV - 1) / (2 * FS_YV), g.nzp, nb);
    fs_dispatch(py.n1, py.n2, py.st, [&](auto a, auto b, auto c) {
      launch(st, gr, FS_YV * std::max(py.n1, py.n2), 0, k4_fwd_y<decltype(a)::value, decltype(b)::value,
             decltype(c)::value>, g, py.n1, py.n2, twy + py.tw4_off, P, M);
    });
    ++ctx->nlaunch;
  } else {
    const int txf = pick_txf(g.Nx);
    const size_t sm_y = sizeof(real2) * (size_t)(txf / 2) * g.Ny * 2;
    for (int b = 0; b < nb; ++b) {
      launch(st, dim3(g.Nx / txf, g.nzp), FFT_THREADS, sm_y, k_fwd_y, g, txf, py, twy, phys[b], mids[b]);
      ++ctx->nlaunch;
    }
  }
  if (px.n1) {
    const int rp = fs_rows(px.n1, px.n2);
    const dim3 gr((unsigned)((nrows + 2 * rp - 1) / (2 * rp)), nb);
    fs_dispatch(px.n1, px.n2, px.st, [&](auto a, auto b, auto c) {
      launch(st, gr, FS_THREADS, 0, k4_fwd_x<decltype(a)::value, decltype(b)::value, decltype(c)::value>, g, px.n1,
             px.n2, nrows, tw + px.tw4_off, MC, Sp);
    });
    ++ctx->nlaunch;
  } else {
    const int rp = pick_rp(g.Nx);
    const size_t sm_x = sizeof(real2) * (size_t)rp * g.Nx * 2;
    for (int b = 0; b < nb; ++b) {
      launch(st, (unsigned)((nrows + 2 * rp - 1) / (2 * rp)), FFT_THREADS, sm_x, k_fwd_x, g, rp, nrows, px, tw,
             mids[b], spec[b]);
      ++ctx->nlaunch;
    }
  }
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

// the inverse x pass of nb arrays (S.op, for SPEC_PAIR
// their x derivatives into mids and their y derivatives into ymids)
void inv_x_pass(pmpic_ctx* ctx, int nb, const SpecIn<real>& S, real* const* mids, real* const* ymids,
                const real2* tw) {
  const Geom& g = ctx->g;
  const FftPlan& px = ctx->plan_x;
  cudaStream_t st = ctx->stream;
  const int64_t nrows = (int64_t)g.nzp * g.sy;
  if (px.n1) {
    Arr6<real> M{}, D{};
    for (int b = 0; b < nb; ++b) {
      M.p[b] = mids[b];
      if (ymids) D.p[b] = ymids[b];
    }
    const int rp = fs_rows(px.n1, px.n2);
    const dim3 gr((unsigned)((nrows + 2 * rp - 1) / (2 * rp)), nb);
    const size_t sm = sizeof(real2) * (size_t)rp * px.n1 * (px.n2 + 1) * (S.op == SPEC_PAIR ? 2 : 1);
    fs_dispatch(px.n1, px.n2, px.st, [&](auto a, auto b, auto c) {
      constexpr int A = decltype(a)::value, B = decltype(b)::value;
      constexpr bool C = decltype(c)::value;
      auto go = [&](auto kern) {
        launch(st, gr, FS_THREADS, sm, kern, g, px.n1, px.n2, nrows, tw + px.tw4_off, S, M, D);
      };
      switch (S.op) {
        case SPEC_PAIR: go(k4_inv_x<A, B, C, SPEC_PAIR>); break;
        default: go(k4_inv_x<A, B, C, SPEC_PLAIN>); break;
      }
    });
    ++ctx->nlaunch;
    return;
  }
  const int rp = pick_rp(g.Nx);
  const size_t sm = sizeof(real2) * (size_t)rp * g.Nx * 2;
  const unsigned nblk = (unsigned)((nrows + 2 * rp - 1) / (2 * rp));
  for (int b = 0; b < nb; ++b) {
    auto go = [&](auto kern, real* mid) {
      launch(st, nblk, FFT_THREADS, sm, kern, g, rp, nrows, px, tw, mid, S, b);
      ++ctx->nlaunch;
    };
    switch (S.op) {
      case SPEC_PAIR:
        go(k_inv_x<SPEC_DX>, mids[b]);
        go(k_inv_x<SPEC_DY>, ymids[b]);
        break;
      default: go(k_inv_x<SPEC_PLAIN>, mids[b]); break;
    }
  }
}
// one Stockham inverse y pass
void inv_y_generic(pmpic_ctx* ctx, const real* mid, real* phys, const real2* twy,
                   const PhysOut<real>& E) {
  const Geom& g = ctx->g;
  const int txf = pick_txf(g.Nx);
  const size_t half = (size_t)g.Ny / 2 + 1;
  const size_t sm = sizeof(real2) * std::max((size_t)(txf / 2) * g.Ny * 2, (size_t)(txf / 2) * g.Ny + txf * half);
  launch(ctx->stream, dim3(g.Nx / txf, g.nzp), FFT_THREADS, sm, k_inv_y, g, txf, ctx->plan_y, twy, mid, phys, E);
  ++ctx->nlaunch;
}

// x then y pass of nb arrays (1..6), the input operator S.op applied on the way
int fft_inverse_impl(pmpic_ctx* ctx, int nb, const SpecIn<real>& S, real* const* phys, real* const* mids,
                     const real2* tw) {
  TimerScope ts(ctx, T_FFTI);
  const Geom& g = ctx->g;
  const FftPlan& py = ctx->plan_y;
  const real2* twy = tw + ctx->ftw_off_y;
  Arr6<const real> M{};
  Arr6<real> P{};
  for (int b = 0; b < nb; ++b) {
    M.p[b] = mids[b];
    P.p[b] = phys[b];
  }
  inv_x_pass(ctx, nb, S, mids, nullptr, tw);
  if (py.n1) {
    const dim3 gr((g.Nx + 2 * FS_YV - 1) / (2 * FS_YV), g.nzp, nb);
    fs_dispatch(py.n1, py.n2, py.st, [&](auto a, auto b, auto c) {
      launch(ctx->stream, gr, FS_YV * std::max(py.n1, py.n2), 0, k4_inv_y<decltype(a)::value, decltype(b)::value,
             decltype(c)::value>, g, py.n1, py.n2, twy + py.tw4_off, M, P);
    });
    ++ctx->nlaunch;
  } else {
    for (int b = 0; b < nb; ++b) inv_y_generic(ctx, mids[b], phys[b], twy, PhysOut<real>{});
  }
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

// The eight inverse transforms of vorticity_tendency.F90:147-265 and its
// products: S.x are the spectra of b, u, v, w, G the grids p, q, r and dp, dq,
// dr, mids eight scratch arrays, work three grids.
int fft_tendency_impl(pmpic_ctx* ctx, const SpecIn<real>& S, const real* const* pqr, real* const* dpqr,
                      real* const* mids, real* const* work, const real2* tw) {
  TimerScope ts(ctx, T_FFTI);
  const Geom& g = ctx->g;
  const FftPlan& py = ctx->plan_y;
  const real2* twy = tw + ctx->ftw_off_y;
  inv_x_pass(ctx, 4, S, mids, mids + 4, tw);  // the x, then the y derivatives of b, u, v, w
  const real *bx = mids[0], *ux = mids[1], *vx = mids[2], *wx = mids[3];
  const real *by = mids[4], *uy = mids[5], *vy = mids[6], *wy = mids[7];
  if (py.n1) {
    VtArgs V{{by, ux, uy, wx, bx, vx, vy, wy}, pqr[0], pqr[1], pqr[2], dpqr[0], dpqr[1], dpqr[2], work[0], work[1]};
    const dim3 gr((g.Nx + 2 * FS_YV - 1) / (2 * FS_YV), g.nzp);
    const size_t sm = sizeof(real2) * 2 * FS_YV * (size_t)(py.n1 * (py.n2 + 1) + 1);
    fs_dispatch(py.n1, py.n2, py.st, [&](auto a, auto b, auto c) {
      launch(ctx->stream, gr, FS_YV * std::max(py.n1, py.n2), sm, k4_vt_y<decltype(a)::value, decltype(b)::value,
             decltype(c)::value>,  g, py.n1, py.n2, twy + py.tw4_off, V);
    });
    ++ctx->nlaunch;
    PMPIC_CUDA(cudaGetLastError());
    return 0;
  }
  const real *P = pqr[0], *Q = pqr[1], *R = pqr[2];
  real *DP = dpqr[0], *DQ = dpqr[1], *DR = dpqr[2], *dudx = work[0], *dwdx = work[1], *dvdy = work[2];
  auto epi = [](int op, int store, real* o, const real* a, const real* c) {
    PhysOut<real> E;
    E.op = op;
    E.store = store;
    E.o = o;
    E.in[0] = a;
    E.in[1] = c;
    return E;
  };
  auto y = [&](const real* mid, real* phys, const PhysOut<real>& E) {
    inv_y_generic(ctx, mid, phys, twy, E);
  };
  y(by, DP, PhysOut<real>{});
  y(ux, dudx, epi(PHYS_ADD_MUL, 1, DP, P, nullptr));
  y(uy, nullptr, epi(PHYS_ADD_MUL, 0, DP, Q, nullptr));
  y(wx, dwdx, epi(PHYS_ADD_MUL_SUM, 1, DP, R, Q));
  y(bx, DQ, PhysOut<real>{});
  y(vx, nullptr, epi(PHYS_NEG_ADD_MUL, 0, DQ, P, nullptr));
  y(vy, dvdy, epi(PHYS_ADD_MUL, 1, DQ, Q, nullptr));
  PhysOut<real> last = epi(PHYS_DQ_DR, 0, DQ, R, P);
  last.o2 = DR;
  last.in[2] = Q;
  last.in[3] = dwdx;
  last.in[4] = dudx;
  last.in[5] = dvdy;
  y(wy, nullptr, last);
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

// shared-memory limits of the kernels with dynamic shared memory that the
// context's lengths use (a property of each function on the current device)
cudaError_t fft_attributes(const FftPlan& px, const FftPlan& py) {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto kern) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  };
  if (px.n1) {
    fs_dispatch(px.n1, px.n2, px.st, [&](auto a, auto b, auto c) {
      set(k4_inv_x<decltype(a)::value, decltype(b)::value, decltype(c)::value, SPEC_PAIR>);
    });
  } else {
    set(k_fwd_x);
    set(k_inv_x<SPEC_PLAIN>);
    set(k_inv_x<SPEC_DX>);
    set(k_inv_x<SPEC_DY>);
  }
  if (py.n1) {
    fs_dispatch(py.n1, py.n2, py.st, [&](auto a, auto b, auto c) {
      set(k4_vt_y<decltype(a)::value, decltype(b)::value, decltype(c)::value>);
    });
  } else {
    set(k_fwd_y);
    set(k_inv_y);
  }
  return e;
}
