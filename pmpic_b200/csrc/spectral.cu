// spectral.cu -- semi-spectral operators and the vort2vel / vorticity_tendency
// pipelines on the B200.
//
// Restates model_core/src/fft/fft_ops.F90 (wavenumbers :111-140, filter
// :176-197, diffx :204-302, diffy :305-401, diffz :419-483, laplinv :505-601,
// tridiagonal :620-656) for one GPU, plus the spectral parts of
// components/vort2vel/src/vort2vel.F90:139-320 and
// components/vorticity_tendency/src/vorticity_tendency.F90:147-265.
//
// Spectral arrays are (Nz+1) x (Ny+2) x (Nx+2), x' fastest; a column is one
// (j', i') pair over all z.  The operators as the C ABI offers them run one
// thread per element or, the compact z operators, one per column, with the
// reference's recurrence and arithmetic (no FMA contraction), so that they
// reproduce the CPU results bit for bit on identical inputs; the inversion's
// spectral part is one kernel (spectral_impl.cuh: k_invert).
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "common.cuh"

namespace pmpic {

namespace {

inline unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

// mean flow of the zero mode (vort2vel.F90:230-241): the trapezoid integral
// and the reference's average (`1./nz` in REAL(4), 0.5*ubar(nz) added to every
// element before the sum), both by one thread in order.
// d, e: the zero-mode values of each level.  The columns pass through shared
// memory ZM_L levels at a time, so that a box of any depth runs; one of more
// levels keeps the integrals in zb in between.
constexpr int ZM_L = 1024;
__global__ void __launch_bounds__(256) k_zmode(Geom g, const double* __restrict__ d, const double* __restrict__ e,
                                               double* zb) {
  PDL_WAIT();
  __shared__ double es[ZM_L + 1], ds[ZM_L + 1], us[ZM_L], vs[ZM_L], avg[2];
  const int nz = g.nzp, t = threadIdx.x;
  const bool deep = nz > ZM_L;
  double* ubar = zb;
  double* vbar = zb + nz;
  const double dz = g.dz;
  double u = 0, v = 0;
  for (int k0 = 0; k0 < nz; k0 += ZM_L) {
    const int n = min(ZM_L, nz - k0);
    for (int i = t; i < min(n + 1, nz - k0); i += 256) {
      es[i] = e[k0 + i];
      ds[i] = d[k0 + i];
    }
    __syncthreads();
    if (t == 0) {
      for (int i = 0; i < n; ++i) {
        us[i] = u;
        vs[i] = v;
        if (k0 + i < nz - 1) {
          u = u + dz / 2. * (es[i] + es[i + 1]);
          v = v - dz / 2. * (ds[i] + ds[i + 1]);
        }
      }
    }
    __syncthreads();
    for (int i = t; deep && i < n; i += 256) {
      ubar[k0 + i] = us[i];
      vbar[k0 + i] = vs[i];
    }
  }
  const double inz = (double)(1.0f / (float)nz);
  double su = 0.0, sv = 0.0;
  for (int k0 = 0; k0 < nz - 1; k0 += ZM_L) {
    const int n = min(ZM_L, nz - 1 - k0);
    if (deep) {
      __syncthreads();
      for (int i = t; i < n; i += 256) {
        us[i] = ubar[k0 + i];
        vs[i] = vbar[k0 + i];
      }
      __syncthreads();
    }
    if (t == 0) {
      for (int i = 0; i < n; ++i) {
        su = su + (us[i] + f4(0.5f) * u);
        sv = sv + (vs[i] + f4(0.5f) * v);
      }
    }
  }
  if (t == 0) {
    avg[0] = inz * su;
    avg[1] = inz * sv;
  }
  __syncthreads();
  for (int k = t; k < nz; k += 256) {
    ubar[k] = (deep ? ubar[k] : us[k]) - avg[0];
    vbar[k] = (deep ? vbar[k] : vs[k]) - avg[1];
  }
}

// FP64 horizontal sums of two FP32 grids per level, in one fixed order: the
// zero modes (kx = ky = 0) of their unscaled forward transforms, kept in FP64
// by the mixed-precision form
__global__ void __launch_bounds__(256) k_hsum2(Geom g, const float* __restrict__ p, const float* __restrict__ q,
                                               double* __restrict__ hs) {
  PDL_WAIT();
  __shared__ double sp[256], sq[256];
  const int k = blockIdx.x;
  const int64_t m = (int64_t)g.Ny * g.Nx;
  const float* P = p + (size_t)k * m;
  const float* Q = q + (size_t)k * m;
  double a = 0.0, b = 0.0;
  // (loads of eight terms in flight, added in the one order)
  constexpr int U = 8;
  for (int64_t e0 = threadIdx.x; e0 < m; e0 += 256 * U) {
    float pv[U], qv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t e = e0 + 256 * u;
      pv[u] = e < m ? P[e] : 0.f;
      qv[u] = e < m ? Q[e] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e0 + 256 * u < m) {
        a += (double)pv[u];
        b += (double)qv[u];
      }
  }
  sp[threadIdx.x] = a;
  sq[threadIdx.x] = b;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sp[threadIdx.x] += sp[threadIdx.x + s];
      sq[threadIdx.x] += sq[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    hs[k] = sp[0];
    hs[g.nzp + k] = sq[0];
  }
}

// ---- elementwise spectral operators --------------------------------------------
// The wavenumber tables are laid out like a spectral level, but kx depends on
// the x index ip alone and ky on the row jp alone: kx is read from row 0
// (kx[ip]) and ky from column 0 (ky[jp * sx]), the same values.
// diffx (fft_ops.F90:266-295): out(i) = -in(i+1) kx, out(i+1) = in(i) kx
__device__ __forceinline__ double dx_of(const double* in, int64_t e, int ip, const double* kx) {
  return (ip & 1) == 0 ? (-1.0 * in[e + 1]) * kx[ip] : in[e - 1] * kx[ip];
}
// diffy (fft_ops.F90:366-394)
__device__ __forceinline__ double dy_of(const double* in, int64_t e, int jp, int sx, const double* ky) {
  return (jp & 1) == 0 ? (-1.0 * in[e + sx]) * ky[jp * sx] : in[e - sx] * ky[jp * sx];
}

struct EwIdx {
  int64_t e;
  int col, ip, jp, k;
};
__device__ __forceinline__ bool ew_index(const Geom& g, EwIdx& x) {
  int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= g.nspec) return false;
  int cols = g.sx * g.sy;
  x.e = e;
  x.k = (int)(e / cols);
  x.col = (int)(e - (int64_t)x.k * cols);
  x.jp = x.col / g.sx;
  x.ip = x.col - x.jp * g.sx;
  return true;
}

__global__ void k_diffx(Geom g, const double* __restrict__ in, double* __restrict__ out, const double* __restrict__ kx) {
  PDL_WAIT();
  EwIdx x;
  if (!ew_index(g, x)) return;
  out[x.e] = dx_of(in, x.e, x.ip, kx);
}
__global__ void k_diffy(Geom g, const double* __restrict__ in, double* __restrict__ out, const double* __restrict__ ky) {
  PDL_WAIT();
  EwIdx x;
  if (!ew_index(g, x)) return;
  out[x.e] = dy_of(in, x.e, x.jp, g.sx, ky);
}
__global__ void k_filter(Geom g, const double* __restrict__ in, double* __restrict__ out,
                         const double* __restrict__ filt) {
  PDL_WAIT();
  EwIdx x;
  if (!ew_index(g, x)) return;
  out[x.e] = in[x.e] * filt[x.col];
}

// ---- compact z operators ----------------------------------------------------------
// (the C ABI's diffz and laplinv; the inversion runs them inside k_invert)
// The z recurrences run one thread per spectral column.  The Thomas factors
// (pivots den and ratios cp of fft_ops.F90:620-656) depend only on the level
// and, for laplinv, on the column's wavenumber: they are tables built once at
// set-up that repeat the sequential recurrence exactly; the right-hand side is
// still divided by the pivot, so the results keep the reference's bits.

// diffz (fft_ops.F90:419-483).  The tridiagonal coefficients are the same for
// every column, so the Thomas factors (cp and the pivots) are computed once on
// the host with the reference's arithmetic and passed in.
__global__ void k_diffz(Geom g, const double* __restrict__ f, double* __restrict__ out,
                        const double* __restrict__ bot, const double* __restrict__ top,
                        const double* __restrict__ coef /* a[nz], den[nz], cp[nz] */, double a1) {
  PDL_WAIT();
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int cols = g.sx * g.sy;
  if (col >= cols) return;
  const int nz = g.nzp;
  const uint32_t cs = (uint32_t)cols;  // level offsets fit 32 bits (the spectral grid is < 2^31)
  const double* A = coef;
  const double* DEN = coef + nz;
  const double* CP = coef + 2 * nz;
  const double dz = (double)g.dz;
  const bool bt = bot != nullptr;
  // forward sweep: f'(1) = d(1)/den(1); f'(i) = (d(i) - a(i) f'(i-1)) / den(i).
  // The loads of each batch of ZB levels are issued before its recurrence, so
  // the loop waits on one memory latency per batch, not per level.
  constexpr int ZB = 8;
  double fm = f[col], f0 = f[cs + col];
  double d1 = bt ? f0 / dz - a1 * bot[col] * dz : 0.0;
  double prev = d1 / DEN[0];
  out[col] = prev;
  for (int kb = 1; kb < nz - 1; kb += ZB) {
    double fb[ZB];
#pragma unroll
    for (int u = 0; u < ZB; ++u)
      if (kb + u < nz - 1) fb[u] = f[(uint32_t)(kb + u + 1) * cs + col];
#pragma unroll
    for (int u = 0; u < ZB; ++u) {
      const int k = kb + u;
      if (k >= nz - 1) break;
      double d = (fb[u] - fm) / 2.0 / dz;
      prev = (d - A[k] * prev) / DEN[k];
      out[(uint32_t)k * cs + col] = prev;
      fm = f0;
      f0 = fb[u];
    }
  }
  {
    int k = nz - 1;
    double dn = bt ? -fm / dz + a1 * top[col] * dz : 0.0;  // fm = f(nz-1)
    prev = (dn - A[k] * prev) / DEN[k];
    out[(uint32_t)k * cs + col] = prev;
  }
  // back substitution: f(i) = f(i) - cp(i+1) f(i+1)
  double nxt = prev;
  for (int kb = nz - 2; kb >= 0; kb -= ZB) {
    double ob[ZB];
#pragma unroll
    for (int u = 0; u < ZB; ++u)
      if (kb - u >= 0) ob[u] = out[(uint32_t)(kb - u) * cs + col];
#pragma unroll
    for (int u = 0; u < ZB; ++u) {
      const int k = kb - u;
      if (k < 0) break;
      nxt = ob[u] - CP[k + 1] * nxt;
      out[(uint32_t)k * cs + col] = nxt;
    }
  }
}

// laplinv (fft_ops.F90:505-601), in place, one thread per column; columns with
// k2 == 0 keep their input (:567).  The Thomas factors of a column depend on
// its wavenumber only, shared by the four columns (2a-1..2a, 2b-1..2b) of one
// mode (a, b): tab holds, per boundary form (f0, df0), the pivots and then the
// ratios cp, each [mode][level], built at set-up (laplinv_tables).  That is the
// inversion's order of them; here lanes of neighbouring modes read lines of
// their own ([level][mode], which they shared: 47 -> 48 us at 128^3, 77 -> 85 at
// 256x256x128, 312 -> 308 at 16x16x1000; the call, which copies the spectrum
// both ways, 4.3 and 24 ms with either).
__global__ void k_laplinv(Geom g, double* __restrict__ f, int df0, const double* __restrict__ tab,
                          const double* __restrict__ k2) {
  PDL_WAIT();
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  const int cols = g.sx * g.sy;
  if (col >= cols) return;
  const double kk = k2[col];
  if (kk == 0) return;
  const int nz = g.nzp;
  const int64_t cs = cols;
  const int nmode = (g.sx >> 1) * (g.sy >> 1);
  const int jp = col / g.sx, ip = col - jp * g.sx;
  const double* __restrict__ DEN = tab + ((size_t)(2 * df0) * nmode + (jp >> 1) * (g.sx >> 1) + (ip >> 1)) * nz;
  const double* __restrict__ CP = DEN + (size_t)nz * nmode;
  const double f16 = (double)f4div(1.f, 6.f), f13 = (double)f4div(1.f, 3.f), f112 = (double)f4div(1.f, 12.f), f56 = (double)f4div(5.f, 6.f);
  const double dz = (double)g.dz;
  const double idz2 = 1.0 / dz / dz;
  const double ai = idz2 - f112 * kk;
  double an;
  double fm, f0, fp;
  f0 = f[col];
  fp = f[cs + col];
  double d;
  if (!df0) {
    d = 0.0;
    an = 0.0;
  } else {
    d = f13 * f0 + f16 * fp;
    an = idz2 - f16 * kk;
  }
  // tridiagonal (fft_ops.F90:620-656) with the tabulated factors
  double prev = d / DEN[0];
  f[col] = prev;
  // loads of each batch of ZB levels first, then its recurrence (one memory
  // latency per batch); the batch reads f above the levels it overwrites
  constexpr int ZB = 4;
  for (int kb = 1; kb < nz; kb += ZB) {
    double fb[ZB], db[ZB];
#pragma unroll
    for (int u = 0; u < ZB; ++u) {
      if (kb + u < nz - 1) fb[u] = f[(int64_t)(kb + u + 1) * cs + col];
      if (kb + u < nz) db[u] = DEN[kb + u];
    }
#pragma unroll
    for (int u = 0; u < ZB; ++u) {
      const int k = kb + u;
      if (k >= nz) break;
      fm = f0;
      f0 = fp;
      double a;
      if (k < nz - 1) {
        fp = fb[u];
        a = ai;
        d = f112 * fm + f56 * f0 + f112 * fp;
      } else {
        a = an;
        d = df0 ? f13 * f0 + f16 * fm : 0.0;
      }
      prev = (d - a * prev) / db[u];
      f[(int64_t)k * cs + col] = prev;
    }
  }
  double nxt = prev;
  for (int kb = nz - 2; kb >= 0; kb -= ZB) {
    double fb[ZB], cb[ZB];
#pragma unroll
    for (int u = 0; u < ZB; ++u)
      if (kb - u >= 0) {
        fb[u] = f[(int64_t)(kb - u) * cs + col];
        cb[u] = CP[kb - u + 1];
      }
#pragma unroll
    for (int u = 0; u < ZB; ++u) {
      const int k = kb - u;
      if (k < 0) break;
      nxt = fb[u] - cb[u] * nxt;
      f[(int64_t)k * cs + col] = nxt;
    }
  }
}

// dt rule (vort2vel.F90:329-372, vorticity_tendency.F90:277-313), one thread
__global__ void k_dt_velocity(Geom g, DevInfo* info, double dtmax) {
  PDL_WAIT();
  double umax = sqrt(info->umax2), vmax = sqrt(info->vmax2), wmax = sqrt(info->wmax2);
  if (umax == 0) umax = f4(1.E-15f);
  if (vmax == 0) vmax = f4(1.E-15f);
  if (wmax == 0) wmax = f4(1.E-15f);
  double Lx = (double)g.Nx * g.dx, Ly = (double)g.Ny * g.dy, Lz = (double)g.nzp * g.dz;
  double dtv = fmin(Lx / umax, fmin(Ly / vmax, Lz / wmax));
  if (dtmax > dtv) {
    info->dtm = dtv;
    info->limiter = 1;
  } else {
    info->dtm = dtmax;
    info->limiter = 0;
  }
}
__global__ void k_dt_vorticity(DevInfo* info, double prefactor, double dtmax) {
  PDL_WAIT();
  double omax = sqrt(info->omax2);
  double dtw = (omax > 0.) ? prefactor / omax : dtmax;
  if (info->dtm > dtw) {
    info->dtm = dtw;
    info->limiter = 2;
  }
}

}  // namespace

// Host-computed Thomas factors of diffz (no bot/top, and bot/top variants).
int diffz_coef(pmpic_ctx* ctx, bool bt, std::vector<double>& out) {
  const int nz = ctx->g.nzp;
  const double a0 = 0., b0 = 1., c0 = 0.;
  const double a1 = f4div(1.f, 6.f), b1 = f4div(2.f, 3.f), c1 = f4div(1.f, 6.f);
  const double an = 0., bn = 1., cn = 0.;
  const double al = f4div(1.f, 3.f), cl = f4div(1.f, 3.f);
  std::vector<double> A(nz), B(nz), C(nz);
  A[0] = a0; B[0] = b0; C[0] = c0;
  for (int k = 1; k < nz - 1; ++k) { A[k] = a1; B[k] = b1; C[k] = c1; }
  A[nz - 1] = an; B[nz - 1] = bn; C[nz - 1] = cn;
  if (bt) { C[0] = cl; A[nz - 1] = al; }
  out.assign(3 * nz, 0.0);
  double den = B[0];
  out[nz + 0] = den;
  for (int i = 1; i < nz; ++i) {
    double cp = C[i - 1] / den;
    den = B[i] - A[i] * cp;
    if (den == 0) return set_error(ctx, PMPIC_ERR_ZERO_PIVOT, "zero pivot in tridiagonal solver (diffz)");
    out[2 * nz + i] = cp;
    out[nz + i] = den;
  }
  for (int i = 0; i < nz; ++i) out[i] = A[i];
  return 0;
}


// The Thomas factors of laplinv (fft_ops.F90:505-601, :620-656) per boundary
// form, level and wavenumber mode (a, b), from the k2 of the mode's columns:
// the pivots den(k) and the ratios cp(k) = c(k-1) / den(k-1) of the
// sequential recurrence, with the coefficients and the operation order of
// k_laplinv (FP64: the same IEEE operations, so the device's FP64 solve keeps
// its bits; FP32 form: 1/den and cp rounded to FP32).  Layout per form:
// den[nmodes][nz], then cp[nmodes][nz]: a column's recurrence reads its own
// lines one after the other.  A zero pivot is the reference's
// abort (:642-645).
int laplinv_tables(pmpic_ctx* ctx, const double* k2cols) {
  const Geom& g = ctx->g;
  const int nz = g.nzp, mx = g.sx / 2, my = g.sy / 2, nmode = mx * my;
  const double f16 = f4div(1.f, 6.f), f13 = f4div(1.f, 3.f), f112 = f4div(1.f, 12.f), f56 = f4div(5.f, 6.f);
  const double dz = g.dz;
  const double i2dz2 = 2.0 / dz / dz, idz2 = 1.0 / dz / dz;
  const size_t per_form = 2 * (size_t)nz * nmode;
  std::vector<double> tab(2 * per_form, 0.0);
  for (int form = 0; form < 2; ++form) {
    double* DEN = tab.data() + form * per_form;
    double* CP = DEN + (size_t)nz * nmode;
    for (int b = 0; b < my; ++b)
      for (int a = 0; a < mx; ++a) {
        const int m = b * mx + a;
        const double kk = k2cols[(size_t)(2 * b) * g.sx + 2 * a];
        const double ai = idz2 - f112 * kk, bi = -i2dz2 - f56 * kk, ci = idz2 - f112 * kk;
        double b1, c1, an, bn;
        if (!form) {
          b1 = 1.0; c1 = 0.0; an = 0.0; bn = 1.0;
        } else {
          b1 = -idz2 - f13 * kk;
          c1 = idz2 - f16 * kk;
          an = idz2 - f16 * kk;
          bn = -idz2 - f13 * kk;
        }
        double den = b1, cprev = c1;
        DEN[(size_t)m * nz] = den;
        for (int k = 1; k < nz; ++k) {
          const double ak = k < nz - 1 ? ai : an, bk = k < nz - 1 ? bi : bn, ck = k < nz - 1 ? ci : 0.0;
          const double cp = cprev / den;
          den = bk - ak * cp;
          if (den == 0 && kk != 0)
            return set_error(ctx, PMPIC_ERR_ZERO_PIVOT, "zero pivot in tridiagonal solver (laplinv)");
          CP[(size_t)m * nz + k] = cp;
          DEN[(size_t)m * nz + k] = den;
          cprev = ck;
        }
      }
  }
  if (!ctx->mixed) {
    PMPIC_CUDA(cudaMalloc(&ctx->lapcp, sizeof(double) * tab.size()));
    PMPIC_CUDA(cudaMemcpy(ctx->lapcp, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice));
    return 0;
  }
  std::vector<float> t32(tab.size());
  for (int form = 0; form < 2; ++form)
    for (size_t i = 0; i < per_form; ++i) {
      const size_t e = form * per_form + i;
      t32[e] = i < (size_t)nz * nmode ? (float)(1.0 / tab[e]) : (float)tab[e];
    }
  PMPIC_CUDA(cudaMalloc(&ctx->lapcp, sizeof(float) * t32.size()));
  PMPIC_CUDA(cudaMemcpy(ctx->lapcp, t32.data(), sizeof(float) * t32.size(), cudaMemcpyHostToDevice));
  return 0;
}

// a table of the inversion's recurrences: reciprocal pivots (FP64: with the
// residual rl of the rounded reciprocal) and ratios cp, level by level
template <class R>
struct ZTab {
  const R *r, *rl, *cp;
};
// rh = 1 / den rounded, rl = its residual: n rh + n rl is n / den before rounding
__global__ void k_recip(int64_t n, const double* __restrict__ den, double* __restrict__ rh, double* __restrict__ rl) {
  PDL_WAIT();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double d = den[i], h = 1.0 / d;
  rh[i] = h;
  rl[i] = __dmul_rn(__fma_rn(-d, h, 1.0), h);
}

namespace f64 {
using real = double;
inline const double* tab_kx(pmpic_ctx* c) { return c->kx; }
inline const double* tab_ky(pmpic_ctx* c) { return c->ky; }
inline const double* tab_k2(pmpic_ctx* c) { return c->k2; }
inline const double* tab_filt(pmpic_ctx* c) { return c->filt; }
inline const double* diffz_tab(pmpic_ctx* c, int which) { return c->sscratch + c->g.nspec + which * 3 * c->g.nzp; }
// ctx->zrec: per diffz form, then per laplinv form, rh and rl
inline ZTab<double> dz_tab(pmpic_ctx* c, int which) {
  const int nz = c->g.nzp;
  const double* r = c->zrec + which * 2 * nz;
  return {r, r + nz, diffz_tab(c, which) + 2 * nz};
}
inline ZTab<double> lap_tab(pmpic_ctx* c, int form) {
  const int64_t n = (int64_t)(c->g.sx >> 1) * (c->g.sy >> 1) * c->g.nzp;
  const double* r = c->zrec + 4 * c->g.nzp + form * 2 * n;
  return {r, r + n, c->lapcp + (2 * form + 1) * n};
}
// the mean flow (vort2vel.F90:230-241) comes from the zero modes of the
// corrected spectra, inside k_invert
inline int zero_mode(pmpic_ctx*) { return 0; }
#include "spectral_impl.cuh"
}  // namespace f64

namespace f32 {
using real = float;
inline const float* tab_kx(pmpic_ctx* c) { return c->wn32; }
inline const float* tab_ky(pmpic_ctx* c) { return c->wn32 + (size_t)c->g.sx * c->g.sy; }
inline const float* tab_k2(pmpic_ctx* c) { return c->wn32 + 2 * (size_t)c->g.sx * c->g.sy; }
inline const float* tab_filt(pmpic_ctx* c) { return c->wn32 + 3 * (size_t)c->g.sx * c->g.sy; }
inline ZTab<float> dz_tab(pmpic_ctx* c, int which) {
  const int nz = c->g.nzp;
  const float* t = c->wn32 + 4 * (size_t)c->g.sx * c->g.sy + which * 3 * nz;
  return {t + nz, nullptr, t + 2 * nz};
}
inline ZTab<float> lap_tab(pmpic_ctx* c, int form) {
  const int64_t n = (int64_t)(c->g.sx >> 1) * (c->g.sy >> 1) * c->g.nzp;
  const float* t = (const float*)c->lapcp + 2 * form * n;
  return {t, nullptr, t + n};
}
// the zero mode stays FP64: horizontal sums of the gridded p and q taken in
// FP64 before the FP32 transforms, then the FP64 mean-flow integral
inline int zero_mode(pmpic_ctx* ctx) {
  const Geom& g = ctx->g;
  launch(ctx->stream, g.nzp, 256, 0, k_hsum2, g, (const float*)ctx->grid[PMPIC_GRID_P],
         (const float*)ctx->grid[PMPIC_GRID_Q], ctx->hsum); ++ctx->nlaunch;
  launch(ctx->stream, 1, 256, 0, k_zmode, g, ctx->hsum, ctx->hsum + g.nzp,
         ctx->zmode); ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}
#include "spectral_impl.cuh"
}  // namespace f32

int spectral_init(pmpic_ctx* ctx) {
  std::vector<double> c0, c1;
  int rc = diffz_coef(ctx, false, c0);
  if (rc) return rc;
  rc = diffz_coef(ctx, true, c1);
  if (rc) return rc;
  const Geom& g = ctx->g;
  double* coef = ctx->sscratch + g.nspec;
  PMPIC_CUDA(cudaMemcpy(coef, c0.data(), sizeof(double) * c0.size(), cudaMemcpyHostToDevice));
  PMPIC_CUDA(cudaMemcpy(coef + 3 * g.nzp, c1.data(), sizeof(double) * c1.size(), cudaMemcpyHostToDevice));
  // FP32 copies of the wavenumber tables and the diffz factors (mixed-precision form)
  const size_t cols = (size_t)g.sx * g.sy;
  std::vector<double> tabs(4 * cols);
  PMPIC_CUDA(cudaMemcpy(tabs.data(), ctx->kx, sizeof(double) * cols, cudaMemcpyDeviceToHost));
  PMPIC_CUDA(cudaMemcpy(tabs.data() + cols, ctx->ky, sizeof(double) * cols, cudaMemcpyDeviceToHost));
  PMPIC_CUDA(cudaMemcpy(tabs.data() + 2 * cols, ctx->k2, sizeof(double) * cols, cudaMemcpyDeviceToHost));
  PMPIC_CUDA(cudaMemcpy(tabs.data() + 3 * cols, ctx->filt, sizeof(double) * cols, cudaMemcpyDeviceToHost));
  std::vector<float> t32(4 * cols + 6 * (size_t)g.nzp);
  for (size_t i = 0; i < 4 * cols; ++i) t32[i] = (float)tabs[i];
  // diffz factors: a, the reciprocal pivots (from the FP64 recurrence), cp
  const int nz = g.nzp;
  for (int v = 0; v < 2; ++v) {
    const std::vector<double>& c = v ? c1 : c0;
    for (int i = 0; i < 3 * nz; ++i)
      t32[4 * cols + (size_t)v * 3 * nz + i] = (i >= nz && i < 2 * nz) ? (float)(1.0 / c[i]) : (float)c[i];
  }
  PMPIC_CUDA(cudaMalloc(&ctx->wn32, sizeof(float) * t32.size()));
  PMPIC_CUDA(cudaMemcpy(ctx->wn32, t32.data(), sizeof(float) * t32.size(), cudaMemcpyHostToDevice));
  PMPIC_CUDA(cudaMalloc(&ctx->hsum, sizeof(double) * 2 * g.nzp));
  if ((rc = laplinv_tables(ctx, tabs.data() + 2 * cols))) return rc;
  if (ctx->mixed) return f32::invert_init(ctx);
  // the FP64 inversion's reciprocal pivots, from the pivots of both solvers
  const int64_t n = (int64_t)(g.sx >> 1) * (g.sy >> 1) * nz;
  PMPIC_CUDA(cudaMalloc(&ctx->zrec, sizeof(double) * (4 * nz + 4 * n)));
  // A copy from pageable memory may return before it has arrived, and the
  // context's stream does not wait for the default stream that makes it.
  PMPIC_CUDA(cudaStreamSynchronize(nullptr));
  for (int v = 0; v < 2; ++v) {
    double* r = ctx->zrec + v * 2 * nz;
    launch(ctx->stream, nblk(nz, 256), 256, 0, k_recip, nz, f64::diffz_tab(ctx, v) + nz, r, r + nz);
    r = ctx->zrec + 4 * nz + v * 2 * n;
    launch(ctx->stream, nblk(n, 256), 256, 0, k_recip, n, ctx->lapcp + 2 * v * n, r, r + n);
    ctx->nlaunch += 2;
  }
  PMPIC_CUDA(cudaStreamSynchronize(ctx->stream));
  return f64::invert_init(ctx);
}

int spec_diffx(pmpic_ctx* ctx, const double* in, double* out) {
  launch(ctx->stream, nblk(ctx->g.nspec, 256), 256, 0, k_diffx, ctx->g, in, out, ctx->kx); ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}
int spec_diffy(pmpic_ctx* ctx, const double* in, double* out) {
  launch(ctx->stream, nblk(ctx->g.nspec, 256), 256, 0, k_diffy, ctx->g, in, out, ctx->ky); ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}
int spec_filter(pmpic_ctx* ctx, const double* in, double* out) {
  launch(ctx->stream, nblk(ctx->g.nspec, 256), 256, 0, k_filter, ctx->g, in, out, ctx->filt); ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}
int spec_diffz(pmpic_ctx* ctx, const double* in, double* out, const double* bot, const double* top) {
  TimerScope ts(ctx, T_DIFFZ);
  const Geom& g = ctx->g;
  launch(ctx->stream, nblk((int64_t)g.sx * g.sy, 128), 128, 0, k_diffz, g, in, out, bot, top, f64::diffz_tab(ctx,
         bot ? 1 : 0), f4div(1.f, 6.f)); ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}
int spec_laplinv(pmpic_ctx* ctx, double* inout, bool df0) {
  TimerScope ts(ctx, T_LAPLINV);
  const Geom& g = ctx->g;
  launch(ctx->stream, nblk((int64_t)g.sx * g.sy, 128), 128, 0, k_laplinv, g, inout, df0 ? 1 : 0, ctx->lapcp,
         ctx->k2); ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

// vort2vel.F90:139-320 and vorticity_tendency.F90:147-265 in the context's precision
int vort2vel_spectral(pmpic_ctx* ctx) {
  return ctx->mixed ? f32::vort2vel_spectral_impl(ctx) : f64::vort2vel_spectral_impl(ctx);
}
int vorticity_tendency_grids(pmpic_ctx* ctx) {
  return ctx->mixed ? f32::vorticity_tendency_grids_impl(ctx) : f64::vorticity_tendency_grids_impl(ctx);
}
// maxima for the dt rule; v2v: velocity limit, vt: vorticity limit
int field_max(pmpic_ctx* ctx, bool v2v, bool vt) {
  int rc = ctx->mixed ? f32::field_max_impl(ctx, v2v, vt) : f64::field_max_impl(ctx, v2v, vt);
  if (rc) return rc;
  if (v2v) {
    launch(ctx->stream, 1, 1, 0, k_dt_velocity, ctx->g, ctx->dinfo, ctx->cfg.dtmax); ++ctx->nlaunch;
  }
  if (vt) {
    launch(ctx->stream, 1, 1, 0, k_dt_vorticity, ctx->dinfo, ctx->cfg.timestep_prefactor,
           ctx->cfg.dtmax); ++ctx->nlaunch;
  }
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace pmpic
