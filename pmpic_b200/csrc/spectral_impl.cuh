// spectral_impl.cuh -- the semi-spectral operators and the vort2vel /
// vorticity_tendency grid pipelines of spectral.cu, written once over the
// scalar type `real` and included by spectral.cu into one namespace per
// precision (FP64 plain path, FP32 mixed-precision form).  The namespace
// provides the tables of its precision (tab_kx, tab_ky, tab_k2, tab_filt,
// lap_tab, dz_tab) and zero_mode.  Not a standalone header.

template <class P>
inline real* RP(P* p) { return reinterpret_cast<real*>(p); }

// ---- the inversion's spectral part (vort2vel.F90:139-320) -----------------------------
// One kernel from the transformed vorticity a, b, c to the corrected, filtered
// vorticity and the velocity spectra.  Every operator on the way acts on a
// column over all levels (the compact z solves, fft_ops.F90:419-601, and d/dz)
// or on a mode's four columns (2i, 2i+1) x (2j, 2j+1) (diffx, diffy, the
// filter).  So a CTA takes a tile of NC columns, NC / 2 of two neighbouring
// rows, keeps three arrays of its columns in shared memory and touches global
// memory to read a, b, c (twice: c's array has to serve lambda first) and to
// write its results once, where separate operators would each stream whole
// spectra.  The recurrences are sequential in z, one thread a column, one
// warp an array; right-hand sides and everything else run on all threads, in
// runs of levels.  What bounds it is the recurrences' latency: four chains of
// nz levels, two dependent operations a level on the FP32 form; on the FP64
// path the quotient by the pivot is n rh + n rl with the two-term reciprocal
// (the division's rounding but for ties that the second term cannot decide),
// four.  Their factors are tables, [mode][level].
// Arithmetic and its order are the separate operators'.
// Measured, ms per step for all that lies between the transforms (ten kernels
// before, and the velocity spectra formed by the inverse x pass): 32^3 FP64
// 0.60 -> 0.11, 96^3 FP32 0.85 -> 0.22, 128^3 FP64 2.0 -> 0.79; 256^3 FP32
// 3.25 -> 3.26, but its inverse transforms 5.0 instead of 6.5.
struct InvArgs {
  real *a, *b, *c;           // in: the spectra; out: corrected and filtered
  real *u, *v, *w;           // out: velocity spectra
  real *us, *vs, *ws;        // and their filtered copies
  const real *kx, *ky, *k2, *filt;
  ZTab<real> lap[2], dz[2];  // per boundary form: laplinv (f0, df0), diffz (without, with boundary values)
  double* zbar;              // mean flow ubar, vbar (FP64 path: written here)
  real* work;                // the columns of the tiles, when they exceed shared memory
  real hdzi;                 // 0.5 / dz (vort2vel.F90:158)
  real rdz, rdzl;            // 1 / dz, two terms (FP64)
  double rdz64;              // 1 / (FP32 dz)
  int nxt;                   // tiles per row pair
};
// n / den with the reciprocal pivot
__device__ __forceinline__ real zquot(real n, real r, real rl) {
  if constexpr (sizeof(real) == 8) return __fma_rn(n, r, __dmul_rn(n, rl));
  else return n * r;
}
__device__ __forceinline__ real zstep(real d, real a, real prev, real r, real rl) {
  if constexpr (sizeof(real) == 8) return zquot(d - a * prev, r, rl);
  else return __fmaf_rn(-a, prev, d) * r;
}
__device__ __forceinline__ real zback(real f, real cp, real nxt) {
  if constexpr (sizeof(real) == 8) return f - cp * nxt;
  else return __fmaf_rn(-cp, nxt, f);
}
// The Thomas recurrence (fft_ops.F90:620-656) of a warp's columns in place:
// right-hand side in, solution out.  X is the lane's column (level stride NC),
// active false for a lane without one; ai the sub-diagonal of the inner
// levels, an the last one's.  The factors of the warp's nm modes (mode m at
// T.x + off + m * nz; only the first nmv exist) come through a ring in shared
// memory, ZCH levels a chunk, three chunks ahead: read as they are needed,
// their latency would bound the recurrence.
constexpr int ZCH = 16, ZRING = 4;
__device__ __forceinline__ void cp_async_z(real* smem, const real* gmem) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (sizeof(real) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem) : "memory");
}
template <int NC, int NM>
__device__ __forceinline__ void thomas(real* X, bool active, int m, int nz, real ai, real an, const ZTab<real>& T,
                                       int64_t off, int nmv, real* ring) {
  constexpr bool D = sizeof(real) == 8;
  constexpr int ZB = 8, SL = ZCH * NM;  // values of a table per chunk
  const int lane = threadIdx.x & 31, nch = (nz + ZCH - 1) / ZCH;
  real* ring2 = ring + ZRING * SL;
  // chunk c of a table (and of the second) into its slot; one group either way
  auto issue = [&](int c, const real* t, const real* t2) {
    if (c >= 0 && c < nch) {
      for (int e = lane; e < SL; e += 32) {
        const int mm = e / ZCH, l = e % ZCH, k = c * ZCH + l;
        if (mm < nmv && k < nz) {
          cp_async_z(ring + (c % ZRING) * SL + l * NM + mm, t + off + (int64_t)mm * nz + k);
          if (D && t2) cp_async_z(ring2 + (c % ZRING) * SL + l * NM + mm, t2 + off + (int64_t)mm * nz + k);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto ready = [&]() {
    asm volatile("cp.async.wait_group 3;\n" ::: "memory");
    __syncwarp();
  };
  // levels 0 .. nz-2 in whole chunks (constant offsets, no bounds: a level is
  // little more than its loads, its two or four dependent operations and its
  // store), then the rest one by one, the last with an
  const int nfull = (nz - 1) / ZCH;
  for (int c = 0; c < 3; ++c) issue(c, T.r, T.rl);
  real prev = real(0);
  for (int c = 0; c < nch; ++c) {
    __syncwarp();  // the slot's last chunk has been read
    issue(c + 3, T.r, T.rl);
    ready();
    const real* r = ring + (c % ZRING) * SL + m;
    const real* rl = ring2 + (c % ZRING) * SL + m;
    real* Xc = X + c * ZCH * NC;
    if (!active) continue;
    if (c < nfull) {
#pragma unroll
      for (int h = 0; h < ZCH; h += ZB) {
        real d[ZB], rr[ZB], ll[ZB];
#pragma unroll
        for (int u = 0; u < ZB; ++u) {
          rr[u] = r[(h + u) * NM];
          ll[u] = D ? rl[(h + u) * NM] : real(0);
          d[u] = Xc[(h + u) * NC];
        }
#pragma unroll
        for (int u = 0; u < ZB; ++u) {  // (level 0: prev is zero)
          prev = zstep(d[u], ai, prev, rr[u], ll[u]);
          Xc[(h + u) * NC] = prev;
        }
      }
    } else {
      for (int l = 0; c * ZCH + l < nz; ++l) {
        prev = zstep(Xc[l * NC], c * ZCH + l == nz - 1 ? an : ai, prev, r[l * NM], D ? rl[l * NM] : real(0));
        Xc[l * NC] = prev;
      }
    }
  }
  // back substitution from level nz-2: f(k) = f(k) - cp(k+1) f(k+1)
  __syncwarp();
  for (int c = nch - 1; c > nch - 4; --c) issue(c, T.cp, nullptr);
  real hi = real(0);  // cp of the level above
  for (int c = nch - 1; c >= 0; --c) {
    __syncwarp();
    issue(c - 3, T.cp, nullptr);
    ready();
    const real* cp = ring + (c % ZRING) * SL + m;
    real* Xc = X + c * ZCH * NC;
    if (!active) continue;
    if (c < nfull) {
#pragma unroll
      for (int h = ZCH - ZB; h >= 0; h -= ZB) {
        real f[ZB], cc[ZB];
#pragma unroll
        for (int u = 0; u < ZB; ++u) {
          cc[u] = cp[(h + u) * NM];
          f[u] = Xc[(h + u) * NC];
        }
#pragma unroll
        for (int u = ZB - 1; u >= 0; --u) {
          prev = zback(f[u], u == ZB - 1 ? hi : cc[u + 1], prev);
          Xc[(h + u) * NC] = prev;
        }
        hi = cc[0];
      }
    } else {
      for (int l = nz - 1 - c * ZCH; l >= 0; --l) {
        if (c * ZCH + l < nz - 1) {
          prev = zback(Xc[l * NC], hi, prev);
          Xc[l * NC] = prev;
        }
        hi = cp[l * NM];
      }
    }
  }
}
// X[k] = f(k, X[k-1], X[k], X[k+1]) for this thread's run of levels k0 .. k1-1,
// in place, given the values either side of the run
template <int NC, class F>
__device__ __forceinline__ void zwalk(real* X, int k0, int k1, real below, real above, F f) {
  if (k0 >= k1) return;
  real fm = below, f0 = X[k0 * NC];
#pragma unroll 4
  for (int k = k0; k < k1; ++k) {
    const real fp = k + 1 < k1 ? X[(k + 1) * NC] : above;
    X[k * NC] = f(k, fm, f0, fp);
    fm = f0;
    f0 = fp;
  }
}

// values of the rings of the three chain warps
template <int NC>
__host__ __device__ constexpr int inv_ring() {
  return 3 * ZRING * ZCH * (NC / 4) * (sizeof(real) == 8 ? 2 : 1);
}
template <int NC, int NT, bool GM>
__global__ void __launch_bounds__(NT, 512 / NT) k_invert(Geom g, const __grid_constant__ InvArgs S) {
  PDL_WAIT();
  constexpr int W = NC / 2, NG = NT / NC;
  extern __shared__ __align__(16) unsigned char zsm[];
  const int nz = g.nzp, sx = g.sx;
  const int64_t cs = (int64_t)sx * g.sy;
  const int col = threadIdx.x % NC, grp = threadIdx.x / NC, warp = threadIdx.x >> 5;
  const int ip = (blockIdx.x % S.nxt) * W + col % W, jp = 2 * (blockIdx.x / S.nxt) + col / W;
  const bool in = ip < sx;
  const int gc = jp * sx + (in ? ip : 0);                 // spectral column
  const int sgx = in ? ((ip & 1) ? -1 : 1) : 0, sgy = (jp & 1) ? -sx : sx;  // to the mode's neighbour columns
  const int cx = col ^ 1, cy = col ^ W;                   // the same in the tile
  constexpr int NM = NC / 4, RING = inv_ring<NC>() / 3;
  real* ring = (real*)zsm + (warp < 3 ? warp : 0) * RING;
  real* F = GM ? S.work + (size_t)blockIdx.x * 3 * nz * NC : (real*)zsm + 3 * RING;  // lambda, then c
  real *A = F + nz * NC, *B = A + nz * NC;
  const real kx = S.kx[in ? ip : 0], ky = S.ky[jp * sx], kk = S.k2[gc];
  const real fl = S.filt[gc], flx = S.filt[gc + sgx], fly = S.filt[gc + sgy];
  const bool solve = in && kk != 0;  // columns with k2 == 0 keep their input (fft_ops.F90:567)
  const int L = (nz + NG - 1) / NG, k0 = min(grp * L, nz), k1 = min(k0 + L, nz);
  const real dz = (real)g.dz;
  const real f16 = (real)f4div(1.f, 6.f), f13 = (real)f4div(1.f, 3.f), f112 = (real)f4div(1.f, 12.f), f56 = (real)f4div(5.f, 6.f);
  const real idz2 = real(1) / dz / dz;
  const real lai = idz2 - f112 * kk, lan = idz2 - f16 * kk;
  // the tile's modes: the first one's factors in the tables, how many exist, and this column's
  const int tx = blockIdx.x % S.nxt;
  const int64_t mode0 = ((int64_t)(blockIdx.x / S.nxt) * (sx >> 1) + tx * (W / 2)) * nz;
  const int nmv = min(NM, (sx >> 1) - tx * (W / 2)), mcol = (col % W) >> 1;
  const bool lanecol = (threadIdx.x & 31) < NC;  // (a chain warp's lane is its column)
  auto dxs = [&](real nb) { return (ip & 1) == 0 ? (real(-1) * nb) * kx : nb * kx; };  // diffx from the neighbour
  auto dys = [&](real nb) { return (jp & 1) == 0 ? (real(-1) * nb) * ky : nb * ky; };
  auto qdz = [&](real n) {  // n / dz
    if constexpr (sizeof(real) == 8) return zquot(n, S.rdz, S.rdzl);
    // FP32: a quotient of two FP32 values is no nearer to a rounding boundary
    // than 2^-49 of itself, so the FP64 product with 1 / dz, off by 2^-52,
    // rounds to the bits of n / dz
    else return (real)((double)n * S.rdz64);
  };
  auto at = [&](int k) { return (int64_t)k * cs + gc; };
  constexpr int LB = 8;  // levels loaded together

  // lambda's right-hand side f = diffx(a) + diffy(b) + dc/dz (2nd order, one-
  // sided at the walls), f(:,1,1) = 0 (vort2vel.F90:158-173)
  if (in) {
    real cm = k0 > 0 ? S.c[at(k0 - 1)] : real(0), c0 = S.c[at(min(k0, nz - 1))];
    for (int kb = k0; kb < k1; kb += LB) {
      real av[LB], bv[LB], cv[LB];
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int k = min(kb + u, nz - 1);
        av[u] = S.a[at(k) + sgx];
        bv[u] = S.b[at(k) + sgy];
        cv[u] = S.c[at(min(k + 1, nz - 1))];
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int k = kb + u;
        if (k >= k1) break;
        real fz;
        if (k == 0) fz = S.hdzi * (real(4) * cv[u] - S.c[at(2)] - real(3) * c0);
        else if (k == nz - 1) fz = S.hdzi * (S.c[at(nz - 3)] + real(3) * c0 - real(4) * cm);
        else fz = (cv[u] - cm) * S.hdzi;
        real v = dxs(av[u]) + dys(bv[u]) + fz;
        if (gc == 0) v = real(0);
        F[k * NC + col] = v;
        cm = c0;
        c0 = cv[u];
      }
    }
  }
  __syncthreads();
  // laplinv's right-hand sides and solves, in place (fft_ops.F90:505-601)
  auto edge = [&](const real* X, real& lo, real& hi) {
    lo = k0 > 0 && k0 < k1 ? X[(k0 - 1) * NC + col] : real(0);
    hi = k1 < nz && k0 < k1 ? X[k1 * NC + col] : real(0);
  };
  auto lap_rhs = [&](real* X, bool df0, real lo, real hi) {
    zwalk<NC>(X + col, k0, k1, lo, hi, [&](int k, real fm, real f0, real fp) {
      if (k == 0) return df0 ? f13 * f0 + f16 * fp : real(0);
      if (k == nz - 1) return df0 ? f13 * f0 + f16 * fm : real(0);
      return f112 * fm + f56 * f0 + f112 * fp;
    });
  };
  real lo, hi;
  edge(F, lo, hi);
  __syncthreads();
  if (solve) lap_rhs(F, true, lo, hi);
  __syncthreads();
  if (warp == 0) thomas<NC, NM>(F + col, lanecol && solve, mcol, nz, lai, lan, S.lap[1], mode0, nmv, ring);
  __syncthreads();
  // lambda filtered; a = a - diffx(lambda), b = b - diffy(lambda) (:179-194)
  if (in) {
    for (int kb = k0; kb < k1; kb += LB) {
      real av[LB], bv[LB];
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int64_t e = at(min(kb + u, nz - 1));
        av[u] = S.a[e];
        bv[u] = S.b[e];
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int k = kb + u;
        if (k >= k1) break;
        A[k * NC + col] = av[u] - dxs(F[k * NC + cx] * flx);
        B[k * NC + col] = bv[u] - dys(F[k * NC + cy] * fly);
      }
    }
  }
  edge(F, lo, hi);
  __syncthreads();
  // c = c - diffz(lambda), c(1,:,:) = 0 (:196-205); meanwhile a and b go out, filtered (:207-218)
  zwalk<NC>(F + col, k0, k1, lo, hi, [&](int k, real fm, real, real fp) {
    return k == 0 || k == nz - 1 ? real(0) : qdz((fp * fl - fm * fl) / real(2));
  });
  __syncthreads();
  if (threadIdx.x < 32) {
    thomas<NC, 1>(F + col, lanecol && in, 0, nz, f16, real(0), S.dz[0], 0, 1, ring);
  } else if (in) {
    for (int k = (threadIdx.x - 32) / NC; k < nz; k += (NT - 32) / NC) {
      S.a[at(k)] = A[k * NC + col] * fl;
      S.b[at(k)] = B[k * NC + col] * fl;
    }
  }
  __syncthreads();
  const real abot = A[col], atop = A[(nz - 1) * NC + col], bbot = B[col], btop = B[(nz - 1) * NC + col];
  if (in) {
    for (int kb = k0; kb < k1; kb += LB) {
      real cv[LB];
#pragma unroll
      for (int u = 0; u < LB; ++u) cv[u] = S.c[at(min(kb + u, nz - 1))];
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int k = kb + u;
        if (k >= k1) break;
        const real c = k == 0 ? real(0) : cv[u] - F[k * NC + col];
        F[k * NC + col] = c;
        S.c[at(k)] = c * fl;
      }
    }
  }
  __syncthreads();
  // the vector potential: laplinv of a, b (f0) and c (df0) (:243-249)
  real loa, hia, lob, hib;
  edge(A, loa, hia);
  edge(B, lob, hib);
  edge(F, lo, hi);
  __syncthreads();
  if (solve) {
    lap_rhs(A, false, loa, hia);
    lap_rhs(B, false, lob, hib);
    lap_rhs(F, true, lo, hi);
  }
  __syncthreads();
  if (warp < 3) {
    thomas<NC, NM>((warp == 0 ? A : (warp == 1 ? B : F)) + col, lanecol && solve, mcol, nz, lai,
                   warp == 2 ? lan : real(0), S.lap[warp == 2], mode0, nmv, ring);
  } else if (sizeof(real) == 8 && blockIdx.x == 0 && threadIdx.x == 96) {
    // mean flow of the zero mode (vort2vel.F90:230-241; k_zmode) from column
    // 0 of the filtered a and b (it keeps its values: k2 == 0)
    const double f0 = S.filt[0], dzd = g.dz;
    double u = 0, v = 0;
    double *ub = S.zbar, *vb = S.zbar + nz;
    ub[0] = vb[0] = 0;
    for (int k = 0; k < nz - 1; ++k) {
      u = u + dzd / 2. * (B[k * NC] * f0 + B[(k + 1) * NC] * f0);
      v = v - dzd / 2. * (A[k * NC] * f0 + A[(k + 1) * NC] * f0);
      ub[k + 1] = u;
      vb[k + 1] = v;
    }
    const double inz = (double)(1.0f / (float)nz);
    double su = 0.0, sv = 0.0;
    for (int k = 0; k < nz - 1; ++k) {
      su = su + (ub[k] + f4(0.5f) * u);
      sv = sv + (vb[k] + f4(0.5f) * v);
    }
    for (int k = 0; k < nz; ++k) {
      ub[k] = ub[k] - inz * su;
      vb[k] = vb[k] - inz * sv;
    }
  }
  __syncthreads();
  // w = dA/dy - dB/dx and its filtered copy (:306-320)
  if (in) {
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      const real w = dys(A[k * NC + cy]) - dxs(B[k * NC + cx]);
      S.w[at(k)] = w;
      S.ws[at(k)] = w * fl;
    }
  }
  edge(A, loa, hia);
  edge(B, lob, hib);
  __syncthreads();
  // dA/dz and dB/dz with boundary values (:255, :284)
  auto dz_rhs = [&](real* X, real lo, real hi, real bot, real top) {
    zwalk<NC>(X + col, k0, k1, lo, hi, [&](int k, real fm, real, real fp) {
      if (k == 0) return qdz(fp) - f16 * bot * dz;
      if (k == nz - 1) return qdz(-fm) + f16 * top * dz;
      return qdz((fp - fm) / real(2));
    });
  };
  dz_rhs(A, loa, hia, abot, atop);
  dz_rhs(B, lob, hib, bbot, btop);
  __syncthreads();
  if (warp < 2) thomas<NC, 1>((warp == 0 ? A : B) + col, lanecol && in, 0, nz, f16, f13, S.dz[1], 0, 1, ring);
  __syncthreads();
  // u = dB/dz - dC/dy, v = dC/dx - dA/dz, the mean flow in mode (0, 0) (:251-302)
  if (in) {
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      real u = B[k * NC + col] - dys(F[k * NC + cy]), v = dxs(F[k * NC + cx]) - A[k * NC + col];
      if (gc == 0) {
        u = (real)S.zbar[k];
        v = (real)S.zbar[nz + k];
      }
      S.u[at(k)] = u;
      S.us[at(k)] = u * fl;
      S.v[at(k)] = v;
      S.vs[at(k)] = v * fl;
    }
  }
}

// Columns per tile and threads per CTA.  A tile costs four recurrences over
// the levels one after the other, whatever its width, so:
// - The narrowest tiles that are on the device all at once, four CTAs of 128
//   threads to an SM at most (96^3 FP32, 32 columns: 0.224 ms a step, 0.332
//   with two CTAs of 256 threads to an SM, and 0.321 for 16 columns, whose 576
//   CTAs nearly fill the 592 places: hence nine tenths of them; 64^3, 8
//   columns: 0.124, 0.197 for 16 and 256 threads).  With a CTA or less per SM,
//   256 threads (32^3 FP64: 0.109 against 0.115).
// - Else the widest tiles of which two share an SM, with 128 threads where
//   three do (128^3 FP64, 16 columns: 0.787 against 0.850) and otherwise 256
//   (256^3 FP32, 32 columns: 3.26 against 3.91, and 3.43 for 16 columns).
// - One CTA per SM, and then global memory in place of shared memory, only for
//   more levels than 8 columns can hold.
struct InvPlan {
  int nc, nt;
  bool gm;
  size_t bytes;  // of shared memory
};
InvPlan invert_plan(const Geom& g) {
  constexpr int64_t SMS = 148, KB = 1024;
  auto ring = [&](int nc) { return (size_t)3 * ZRING * ZCH * (nc / 4) * (sizeof(real) == 8 ? 2 : 1); };
  auto bytes = [&](int nc) { return ((size_t)3 * g.nzp * nc + ring(nc)) * sizeof(real); };
  auto tiles = [&](int nc) { return (int64_t)(g.sy / 2) * ((g.sx + nc / 2 - 1) / (nc / 2)); };
  for (int nc = 8; nc <= 32; nc *= 2) {
    const int64_t places = SMS * min((int64_t)4, 225 * KB / ((int64_t)bytes(nc) + KB));
    if (tiles(nc) * 10 <= places * 9) return InvPlan{nc, tiles(nc) <= SMS ? 256 : 128, false, bytes(nc)};
  }
  int nc = 32;
  while (nc > 8 && (int64_t)bytes(nc) > 112 * KB) nc /= 2;
  if ((int64_t)bytes(nc) > 224 * KB) return InvPlan{nc, 256, true, ring(nc) * sizeof(real)};
  return InvPlan{nc, (int64_t)bytes(nc) <= 74 * KB ? 128 : 256, false, bytes(nc)};
}
template <class F>
void invert_kernel(const InvPlan& p, F&& f) {
  if (p.gm) f(k_invert<8, 256, true>);
  else if (p.nc == 32) f(p.nt == 128 ? k_invert<32, 128, false> : k_invert<32, 256, false>);
  else if (p.nc == 16) f(p.nt == 128 ? k_invert<16, 128, false> : k_invert<16, 256, false>);
  else f(p.nt == 128 ? k_invert<8, 128, false> : k_invert<8, 256, false>);
}
int invert_init(pmpic_ctx* ctx) {
  const Geom& g = ctx->g;
  const InvPlan p = invert_plan(g);
  if (p.gm) {
    const int64_t tiles = (int64_t)(g.sy / 2) * ((g.sx + p.nc / 2 - 1) / (p.nc / 2));
    PMPIC_CUDA(cudaMalloc(&ctx->zwork, sizeof(real) * 3 * (size_t)g.nzp * p.nc * tiles));
    return 0;
  }
  cudaError_t e = cudaSuccess;
  invert_kernel(p, [&](auto k) { e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024); });
  PMPIC_CUDA(e);
  return 0;
}
int invert_launch(pmpic_ctx* ctx, real* a, real* b, real* c, real* u, real* v, real* w) {
  TimerScope ts(ctx, T_LAPLINV);
  const Geom& g = ctx->g;
  const InvPlan p = invert_plan(g);
  InvArgs S{a, b, c, u, v, w, RP(ctx->spec[PMPIC_SPEC_U]), RP(ctx->spec[PMPIC_SPEC_V]), RP(ctx->spec[PMPIC_SPEC_W]),
            tab_kx(ctx), tab_ky(ctx), tab_k2(ctx), tab_filt(ctx), {lap_tab(ctx, 0), lap_tab(ctx, 1)},
            {dz_tab(ctx, 0), dz_tab(ctx, 1)}, ctx->zmode, (real*)ctx->zwork, (real)(f4div(1.f, 2.f) / g.dz)};
  const double r = 1.0 / g.dz;
  S.rdz = (real)r;
  S.rdzl = (real)(std::fma(-g.dz, r, 1.0) * r);
  S.rdz64 = 1.0 / (double)(real)g.dz;
  S.nxt = (g.sx + p.nc / 2 - 1) / (p.nc / 2);
  invert_kernel(p, [&](auto k) { launch(ctx->stream, (unsigned)(S.nxt * (g.sy / 2)), p.nt, p.bytes, k, g, S); });
  ++ctx->nlaunch;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

// a CTA's maximum into *out (one atomic per CTA)
__device__ __forceinline__ void cta_max(real m, double* __restrict__ out) {
  __shared__ real sh[8];
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = fmax(m, sh[w]);
    atomicMax((unsigned long long*)out, __double_as_longlong((double)m));
  }
}
// max of squares over the interior (vort2vel.F90:331-338,
// vorticity_tendency.F90:279-282); non-negative doubles order like their bits
__global__ void k_max_sq3(int64_t n, const real* __restrict__ u, const real* __restrict__ v,
                          const real* __restrict__ w, double* __restrict__ out3) {
  PDL_WAIT();
  real mu = 0, mv = 0, mw = 0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    real a = u[e], b = v[e], c = w[e];
    mu = fmax(mu, a * a);
    mv = fmax(mv, b * b);
    mw = fmax(mw, c * c);
  }
  cta_max(mu, &out3[0]);
  cta_max(mv, &out3[1]);
  cta_max(mw, &out3[2]);
}
__global__ void k_max_vort(int64_t n, const real* __restrict__ p, const real* __restrict__ q,
                           const real* __restrict__ r, double* __restrict__ out) {
  PDL_WAIT();
  real m = 0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    real a = p[e], b = q[e], c = r[e];
    m = fmax(m, a * a + b * b + c * c);
  }
  cta_max(m, out);
}

// vort2vel.F90:139-320 after the three par2grid calls (grids P, Q, R hold the
// gridded vorticity on entry; on exit they hold the corrected, filtered
// vorticity, U, V, W the velocity and u_s, v_s, w_s its filtered spectra).
int vort2vel_spectral_impl(pmpic_ctx* ctx) {
  const Geom& g = ctx->g;
  int rc;
  real *a = RP(ctx->sa), *b = RP(ctx->sb), *c = RP(ctx->sc), *u = RP(ctx->sd), *v = RP(ctx->se), *w = RP(ctx->sf);
  real* const* G = (real* const*)ctx->grid;
  if ((rc = zero_mode(ctx))) return rc;
  // scratch of the transforms: these arrays hold nothing that the inversion
  // reads (the packed gather grids are made afresh before they are used, and
  // their six grids hold three of the arrays: Ny + 2 <= 2 Ny)
  const size_t nmid = (size_t)g.nzp * g.sy * g.Nx;
  real* pk = RP(ctx->gpack);
  real* mids[6] = {RP(ctx->fftmid), RP(ctx->sas), RP(ctx->sbs), pk, pk + nmid, pk + 2 * nmid};
  {
    const real* in[3] = {G[PMPIC_GRID_P], G[PMPIC_GRID_Q], G[PMPIC_GRID_R]};
    real* out[3] = {a, b, c};
    if ((rc = fft_forward(ctx, 3, in, out, mids))) return rc;
  }
  if ((rc = invert_launch(ctx, a, b, c, u, v, w))) return rc;
  // the corrected, filtered vorticity (:207-226) and the velocity (:251-320)
  SpecIn<real> S;
  const real* in[6] = {a, b, c, u, v, w};
  real* out[6] = {G[PMPIC_GRID_P], G[PMPIC_GRID_Q], G[PMPIC_GRID_R], G[PMPIC_GRID_U], G[PMPIC_GRID_V], G[PMPIC_GRID_W]};
  for (int q = 0; q < 6; ++q) S.x[q] = in[q];
  return fft_inverse(ctx, 6, S, out, mids);
}

// vorticity_tendency.F90:147-265 (grid B holds par2grid(btot) on entry).  The
// x pass reads each of the spectra of b, u, v, w once and transforms its two
// derivatives; the y pass forms dp, dq and dr as it transforms them.
int vorticity_tendency_grids_impl(pmpic_ctx* ctx) {
  int rc;
  real* const* G = (real* const*)ctx->grid;
  real* bs = RP(ctx->sbs);
  const real* bg = G[PMPIC_GRID_B];
  real* mid0 = RP(ctx->fftmid);
  if ((rc = fft_forward(ctx, 1, &bg, &bs, &mid0))) return rc;
  SpecIn<real> S;
  S.op = SPEC_PAIR;
  S.x[0] = bs;
  for (int q = 0; q < 3; ++q) S.x[q + 1] = RP(ctx->spec[PMPIC_SPEC_U + q]);
  S.kx = tab_kx(ctx);
  S.ky = tab_ky(ctx);
  const real* pqr[3] = {G[PMPIC_GRID_P], G[PMPIC_GRID_Q], G[PMPIC_GRID_R]};
  real* dpqr[3] = {G[PMPIC_GRID_DP], G[PMPIC_GRID_DQ], G[PMPIC_GRID_DR]};
  real* mids[8] = {mid0, RP(ctx->sas), RP(ctx->sa), RP(ctx->sb), RP(ctx->sc), RP(ctx->sd), RP(ctx->se), RP(ctx->sf)};
  real* work[3] = {RP(ctx->gwork[0]), RP(ctx->gwork[1]), RP(ctx->gwork[2])};
  if ((rc = fft_tendency(ctx, S, pqr, dpqr, mids, work))) return rc;
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

// maxima for the dt rule; v2v: velocity limit, vt: vorticity limit
int field_max_impl(pmpic_ctx* ctx, bool v2v, bool vt) {
  real* const* G = (real* const*)ctx->grid;
  const Geom& g = ctx->g;
  if (v2v) {
    PMPIC_CUDA(cudaMemsetAsync(&ctx->dinfo->umax2, 0, 3 * sizeof(double), ctx->stream));
    launch(ctx->stream, 592, 256, 0, k_max_sq3, g.nphys, G[PMPIC_GRID_U], G[PMPIC_GRID_V], G[PMPIC_GRID_W],
           &ctx->dinfo->umax2); ++ctx->nlaunch;
  }
  if (vt) {
    PMPIC_CUDA(cudaMemsetAsync(&ctx->dinfo->omax2, 0, sizeof(double), ctx->stream));
    launch(ctx->stream, 592, 256, 0, k_max_vort, g.nphys, G[PMPIC_GRID_P], G[PMPIC_GRID_Q], G[PMPIC_GRID_R],
           &ctx->dinfo->omax2); ++ctx->nlaunch;
  }
  PMPIC_CUDA(cudaGetLastError());
  return 0;
}

