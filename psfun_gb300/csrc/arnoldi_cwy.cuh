// arnoldi_cwy.cuh -- a whole Arnoldi solve in one cooperative launch, with two
// grid barriers per step (included by krylov.cu).
//
// Modified Gram-Schmidt (psfun_d_arnoldi.f90:210-214) takes its coefficients
// one after another, h_k = v_k . (w - sum_{j<k} h_j v_j), a grid barrier and a
// reduction each (every second one in k_ar_mgs_sm): ~5 us per pair of vectors
// whatever n is, 38 us per step at n = 10,000 and 65 at n = 86,000.  Written
// out, the same coefficients are
//     h_k = v_k . w - sum_{j<k} (v_k . v_j) h_j,   i.e.  (I + L) h = V^T w
// with L the strictly lower part of V^T V (the compact form of MGS, Swirydowicz,
// Langou, Ananthan, Yang, Thomas, "Low synchronization Gram-Schmidt and
// generalized minimal residual algorithms", 2021): all dots of a step are taken
// at once, together with those of the newest vector v_{i-1} with the others
// (L's next row), and the second barrier sums the norm of the result.  The
// price is one more pass over the basis (the dots for L): 2 n DFMA per vector
// against half a barrier and reduction (~2.5 us), even near n = 740,000.
// What bounds it: at n = 10,000 the two barriers and the chains of dependent
// loads and sums between them (8-12 us per step, 38 before), from n = 90,000
// on the FP64 pipe (6 n i FMA-cycles per step).  Measured per solve, against
// k_ar_mgs_sm: 2-D 5-point, 60 vectors, n = 10,000 1.10 ms (4.79), 90,000 2.16
// (5.30), 262,144 4.23 (6.84), 490,000 6.91 (9.03).
//
// L is at rounding level (1e-16) for an orthogonal basis, so h = r - L r to
// O(L^2), formed in FP32 (it needs as many digits as L^-1 eps has) while
// |L| <= 1e-8, and by forward substitution in FP64 beyond.
//
// A block owns `chunk` rows of every vector.  With VS its rows of the whole
// basis stay in shared memory for the solve (n (nl - 1) <= ~3.5e6 on 152 SMs)
// and each pass reads them from there; otherwise the passes read the basis
// from L2.  A warp owns 32 rt of the block's rows and every kg-th vector, forms
// lane partials of the two dots in FP64 and sums them over the lanes and the
// grid on the integer pipe (fixsum.cuh).
#pragma once

struct CwyPlan : CwyShape {
  bool vs = false;
  size_t smem = 0;
};

constexpr int kCwyMaxNl = 128;
constexpr size_t kCwySmemMax = 220 * 1024;  // leaves the estimate monitors' static shared memory

// 64-bit words of one buffer of grid sums: r and l limbs per vector, the three
// limbs of the norm, the flag.
__host__ __device__ inline int cwy_acc_words(int nl) { return 4 * nl + 8; }

static size_t cwy_smem_bytes(int nl, int chunk, int rt, bool vs) {
  const size_t nrg = (size_t)(chunk + 32 * rt - 1) / (32 * rt);
  size_t d = (size_t)chunk * (vs ? nl : 2) + 4 * (size_t)(nl + 2) + 4 * nrg * nl + 3 * 32;
  return 8 * d + 4 * ((size_t)nl * (nl - 1) / 2 + 2 * (nl + 2)) + 64;
}

// The dots of one warp: its 32 RT rows of w and of the newest vector with the
// vectors kq + 1, kq + 1 + kg, ... (the newest one with w only).
struct CwyDots {
  const double *wl, *vl;
  const int* il;
  long long* part;
  int row, nloc, nv, ew;
};

template <bool VS, int RT>
PSF_DEVINL bool cwy_dots(const CwyDots& d, const double* v1, int64_t ldk, int kq, int kg) {
  const int lane = threadIdx.x & 31;
  double w[RT], x[RT];
#pragma unroll
  for (int q = 0; q < RT; ++q) {
    const bool on = d.row + 32 * q < d.nloc;
    w[q] = on ? d.wl[d.row + 32 * q] : 0.0;
    x[q] = on ? d.vl[d.row + 32 * q] : 0.0;
  }
  bool ok = true;
  auto load = [&](int k, double (&v)[RT]) {
    const double* vk = v1 + (int64_t)(k - 1) * ldk + d.row;
#pragma unroll
    for (int q = 0; q < RT; ++q) v[q] = d.row + 32 * q < d.nloc ? (VS ? vk[32 * q] : __ldcg(vk + 32 * q)) : 0.0;
  };
  auto put = [&](int k, int at, double a, int E) {
    int p[4];
    long long hi, lo;
    ok &= fix96_pieces(a, E, p);
    fix96_warp(p, hi, lo);
    if (lane == 0) {
      d.part[(size_t)(k - 1) * 4 + at] = hi;
      d.part[(size_t)(k - 1) * 4 + at + 1] = lo;
    }
  };
  auto dot = [&](const double (&v)[RT], const double (&u)[RT]) {
    double a = v[0] * u[0];
#pragma unroll
    for (int q = 1; q < RT; ++q) a = fma(v[q], u[q], a);
    return a;
  };
  int k = kq + 1;
  // two vectors at a time: their loads and reductions overlap
  for (; k + kg < d.nv; k += 2 * kg) {
    double va[RT], vb[RT];
    load(k, va);
    load(k + kg, vb);
    const double a0 = dot(va, w), l0 = dot(va, x), a1 = dot(vb, w), l1 = dot(vb, x);
    put(k, 0, a0, d.ew - d.il[k]);
    put(k, 2, l0, 1 - d.il[k] - d.il[d.nv]);
    put(k + kg, 0, a1, d.ew - d.il[k + kg]);
    put(k + kg, 2, l1, 1 - d.il[k + kg] - d.il[d.nv]);
  }
  for (; k < d.nv; k += kg) {
    double va[RT];
    load(k, va);
    const double a0 = dot(va, w), l0 = dot(va, x);
    put(k, 0, a0, d.ew - d.il[k]);
    put(k, 2, l0, 1 - d.il[k] - d.il[d.nv]);
  }
  if (k == d.nv) put(k, 0, dot(x, w), d.ew - d.il[k]);
  return ok;
}

template <bool VS>
__global__ void __launch_bounds__(kCwyThreads, 1) k_ar_cwy(KState st, CsrDev A, double scaling, int chunk, int rt,
                                                              int ew, int monitors, long long* acc_all, double* Lg,
                                                              LzMonitor mon) {
  extern __shared__ __align__(16) double cwy_sm[];
  __shared__ int s_bad, s_slow, s_end;
  KCtrl* c = st.ctrl;
  const int nl = st.nl, G = gridDim.x - monitors, b = blockIdx.x;
  const int t = threadIdx.x, bd = blockDim.x, lane = t & 31, warp = t >> 5;
  const bool lead = t == bd - 32;  // forms beta and s (a lane of the warp with the fewest rows)
  if (b >= G) {
    est_monitor_cta(st, mon, 1, nl + 1, b - G);
    return;
  }
  const int nrg = (chunk + 32 * rt - 1) / (32 * rt);  // row groups, one warp each
  const int kg = (bd >> 5) / nrg;                     // warps that share a row group, by vectors
  double* wl = cwy_sm;                                // the block's rows of w
  double* Vs = wl + chunk;                            // VS: of W_1 .. W_{nl-1}; else of W_{i-1}
  double* ss = Vs + (size_t)chunk * (VS ? nl - 1 : 1);  // s_k (1-based)
  double* rv = ss + nl + 2;                           // r_k, then c_k (0-based)
  double* lv = rv + nl + 2;                           // l_k
  double* hv = lv + nl + 2;                           // h_k
  long long* part = reinterpret_cast<long long*>(hv + nl + 2);  // [row group][k][r hi, r lo, l hi, l lo]
  long long* red3 = part + (size_t)4 * nrg * nl;      // [warp][3]
  float* rf = reinterpret_cast<float*>(red3 + 3 * 32);
  int* il = reinterpret_cast<int*>(rf + nl + 2);      // floor(log2 s_k)
  float* Lf = reinterpret_cast<float*>(il + nl + 2);  // row k (0-based) of L at k (k - 1) / 2
  const int64_t r0 = (int64_t)b * chunk;
  const int nloc = (int)max((int64_t)0, min(r0 + chunk, st.n) - r0);
  const int aw = cwy_acc_words(nl);
  unsigned nb = 0;
  int last = 0;
  const bool zero_x = c->done != 0;
  if (!zero_x) {
    const double* w1 = WAT(st, 1) + r0;
    for (int l = t; l < nloc; l += bd) Vs[l] = w1[l];
    if (t == 0) {
      ss[1] = st.s[1];
      il[1] = ilog2_normal(ss[1]);
      s_bad = s_slow = s_end = 0;
    }
    __syncthreads();
  }
  for (int i = 2; i <= nl && !zero_x; ++i) {
    const int nv = i - 1;
    long long* acc = acc_all + (size_t)(i % 3) * aw;
    const double* vl = VS ? Vs + (size_t)(nv - 1) * chunk : Vs;  // rows of W_{i-1}
    // ---- w = scaling s_{i-1} A W_{i-1} on the block's rows (psfun_d_arnoldi.f90:202).
    // s_{i-1} is formed by one thread meanwhile (sqrt and division: ~1200 clocks).
    {
      const double* __restrict__ x = WAT(st, nv);
      for (int l = t; l < nloc; l += bd) {
        const int kb = A.irp[r0 + l], ke = A.irp[r0 + l + 1];
        double s = 0.0;
        for (int k = kb; k < ke; k += 4) {
          double v[4], xv[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const bool on = k + q < ke;
            v[q] = on ? A.val[k + q] : 0.0;
            xv[q] = on ? __ldcg(x + A.ja[k + q]) : 0.0;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (k + q < ke) s = fma(v[q], xv[q], s);
        }
        wl[l] = s;
      }
      if (b == 0 && t == 0) c->stop_dec = *(volatile int*)&c->stop_req;
      if (i > 2 && lead) {  // the norm of the previous step (every block alike)
        const long long* pn = acc_all + (size_t)((i - 1) % 3) * aw + 4 * nl;
        const long long w0 = ld_relaxed_s64(pn), w1 = ld_relaxed_s64(pn + 1), w2 = ld_relaxed_s64(pn + 2);
        const bool bad = ld_relaxed_s64(pn + 3) != 0;
        const double beta = bad ? __longlong_as_double(0x7ff8000000000000ll) : sqrt(fix144_value(w2, w1, w0, 2 * ew));
        const double s = 1.0 / beta;
        ss[nv] = s;
        il[nv] = ilog2_normal(s);
        if (beta == 0.0) s_end = 1;
        if (b == 0) {
          HAT(st, nv, nv - 1) = beta;
          st.s[nv] = s;
          c->itx = nv - 1;
          if (beta == 0.0) c->breakdown = 1;
          if (st.host_flag) st.host_flag[1] = nv;
          st_release_gpu(&c->pub, nv - 1);
        }
        last = nv - 1;
      }
      __syncthreads();
      if (s_end) {  // h(i-1,i-2) == 0: the solve ends on the invariant subspace
        if (b == 0 && t == 0) c->done = 1;
        break;
      }
      const double f = scaling * ss[nv];
      for (int l = t; l < nloc; l += bd) wl[l] *= f;
      __syncthreads();
    }
    // ---- dots of w and of W_{i-1} with the basis: lane partials over the
    // warp's rows, then the fixed-point sums
    {
      const int rg = warp % nrg, kq = warp / nrg;
      if (kq < kg) {
        bool ok = true;
        const CwyDots d{wl, vl, il, part + (size_t)rg * nl * 4, rg * 32 * rt + lane, nloc, nv, ew};
        const double* v1 = VS ? Vs : WAT(st, 1) + r0;
        const int64_t ldk = VS ? chunk : st.ldv;
        switch (rt) {
          case 1: ok = cwy_dots<VS, 1>(d, v1, ldk, kq, kg); break;
          case 2: ok = cwy_dots<VS, 2>(d, v1, ldk, kq, kg); break;
          case 3: ok = cwy_dots<VS, 3>(d, v1, ldk, kq, kg); break;
          case 4: ok = cwy_dots<VS, 4>(d, v1, ldk, kq, kg); break;
          case 5: ok = cwy_dots<VS, 5>(d, v1, ldk, kq, kg); break;
          case 6: ok = cwy_dots<VS, 6>(d, v1, ldk, kq, kg); break;
          case 7: ok = cwy_dots<VS, 7>(d, v1, ldk, kq, kg); break;
          default: ok = false;  // no plan has more (kCwyMaxRt)
        }
        static_assert(kCwyMaxRt == 7, "one case per row count of a plan");
        if (!ok) s_bad = 1;
      }
      __syncthreads();
      if (t < 2 * nv - 1) {  // t < nv: r of vector t + 1; then l of vector t - nv + 1
        const int k = t < nv ? t : t - nv, sel = t < nv ? 0 : 2;
        long long hi = 0, lo = 0;
        for (int g = 0; g < nrg; ++g) {
          const long long* o = part + ((size_t)g * nl + k) * 4 + sel;
          hi += o[0];
          lo += o[1];
        }
        fix96_carry(hi, lo);
        long long* o = acc + (t < nv ? 0 : 2 * nl) + 2 * k;
        red_add_s64(o, hi);
        red_add_s64(o + 1, lo);
      }
      if (t == 0 && s_bad) red_add_s64(acc + 4 * nl + 3, 1);
    }
    if (!grid_sync_to(&c->bar_count, (++nb) * (unsigned)G, &c->err)) break;
    if (*(volatile int*)&c->stop_dec) {
      if (b == 0 && t == 0) c->done = 1;
      break;
    }
    // ---- h = (I + L)^{-1} r
    const bool bad = ld_relaxed_s64(acc + 4 * nl + 3) != 0;
    if (t < 2 * nv - 1) {
      const bool isr = t < nv;
      const int k = isr ? t : t - nv;
      const long long* o = acc + (isr ? 0 : 2 * nl) + 2 * k;
      const long long hi = ld_relaxed_s64(o), lo = ld_relaxed_s64(o + 1);
      const double sk = ss[k + 1];
      double v = fix96_value(hi, lo, isr ? ew - il[k + 1] : 1 - il[k + 1] - il[nv]) * (isr ? sk : sk * ss[nv]);
      if (bad) v = __longlong_as_double(0x7ff8000000000000ll);
      if (isr) {
        rv[k] = v;
        rf[k] = (float)scale_pow2(v, -ew);  // |r_k| <= ||w|| < 2^ew
      } else {
        lv[k] = v;
        Lf[(size_t)(nv - 1) * (nv - 2) / 2 + k] = (float)v;
        if (b == 0) Lg[(size_t)(nv - 1) * nl + k] = v;
        if (!(fabs(v) <= 1e-8)) s_slow = 1;
      }
    }
    __syncthreads();
    if (!s_slow) {
      // eight lanes per row of L
      for (int k = t >> 3; k < nv; k += bd >> 3) {
        float s = 0.0f;
        const float* row = Lf + (size_t)k * (k - 1) / 2;
        for (int j = t & 7; j < k; j += 8) s = fmaf(row[j], rf[j], s);
        const unsigned m8 = 0xffu << (lane & 24);
        s += __shfl_xor_sync(m8, s, 1);
        s += __shfl_xor_sync(m8, s, 2);
        s += __shfl_xor_sync(m8, s, 4);
        if ((t & 7) == 0) hv[k] = rv[k] - scale_pow2((double)s, ew);
      }
    } else {
      // the basis has lost orthogonality: forward substitution in FP64 (the
      // rows of L before this step's from block 0's copy, this step's from lv)
      if (warp == 0) {
        for (int k = 0; k < nv; ++k) {
          double s = 0.0;
          for (int j = lane; j < k; j += 32)
            s = fma((k == nv - 1) ? lv[j] : __ldcg(Lg + (size_t)k * nl + j), hv[j], s);
          s = warp_sum(s);
          if (lane == 0) hv[k] = rv[k] - s;
          __syncwarp();
        }
      }
    }
    __syncthreads();
    if (t < nv) {
      const double h = hv[t];
      if (b == 0) HAT(st, t + 1, i - 1) = h;
      rv[t] = h * ss[t + 1];  // c_k
    }
    if (b == 0)  // the next step's sums start at zero (no block reads or adds to them before this step's end)
      for (int l = t; l < aw; l += bd) acc_all[(size_t)((i + 1) % 3) * aw + l] = 0;
    __syncthreads();
    // ---- w -= sum_k c_k W_k, the squared norm, W_i to global memory
    {
      double* wo = WAT(st, i) + r0;
      double* vo = (VS && i < nl) ? Vs + (size_t)nv * chunk : nullptr;
      double p = 0.0;
      for (int l = t; l < nloc; l += bd) {
        double w = wl[l];
        int k = 0;
        for (; k + 4 <= nv; k += 4) {
          double v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            v[u] = VS ? Vs[(size_t)(k + u) * chunk + l] : __ldcg(WAT(st, k + u + 1) + r0 + l);
#pragma unroll
          for (int u = 0; u < 4; ++u) w = fma(-rv[k + u], v[u], w);
        }
        for (; k < nv; ++k) w = fma(-rv[k], VS ? Vs[(size_t)k * chunk + l] : __ldcg(WAT(st, k + 1) + r0 + l), w);
        wo[l] = w;
        if (VS) {
          if (vo) vo[l] = w;
        } else {
          Vs[l] = w;  // the rows of W_{i-1}: only this thread read them in this pass
        }
        p = fma(w, w, p);
      }
      long long w3[3];
      const bool ok = fix144_limbs(p, 2 * ew, w3);
      if (!ok) s_bad = 1;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const long long v = warp_sum_s64(w3[q]);
        if (lane == 0) red3[warp * 3 + q] = v;
      }
      __syncthreads();
      if (t == 0) {
        long long q0 = 0, q1 = 0, q2 = 0;
        for (int g = 0; g < (bd >> 5); ++g) {
          q0 += red3[3 * g];
          q1 += red3[3 * g + 1];
          q2 += red3[3 * g + 2];
        }
        fix96_carry(q1, q0);
        fix96_carry(q2, q1);
        red_add_s64(acc + 4 * nl, q0);
        red_add_s64(acc + 4 * nl + 1, q1);
        red_add_s64(acc + 4 * nl + 2, q2);
        if (s_bad) red_add_s64(acc + 4 * nl + 3, 1);
        s_bad = 0;
      }
    }
    if (!grid_sync_to(&c->bar_count, (++nb) * (unsigned)G, &c->err)) break;
    if (i == nl && b == 0 && lead) {  // the last step's norm
      const long long* pn = acc + 4 * nl;
      const double beta = ld_relaxed_s64(pn + 3) != 0
                              ? __longlong_as_double(0x7ff8000000000000ll)
                              : sqrt(fix144_value(ld_relaxed_s64(pn + 2), ld_relaxed_s64(pn + 1), ld_relaxed_s64(pn),
                                                  2 * ew));
      HAT(st, i, i - 1) = beta;
      st.s[i] = 1.0 / beta;
      c->itx = i - 1;
      if (beta == 0.0) c->breakdown = 1;
      if (st.host_flag) st.host_flag[1] = i;
      st_release_gpu(&c->pub, i - 1);
      last = i - 1;
    }
  }
  if (b == 0 && lead) st_release_gpu(&c->steps_end, last + 1);
}

// Grid, rows per block and shared memory of k_ar_cwy, or none: Krylov
// dimension above kCwyMaxNl, a row above 64 entries (one thread per row), n of
// 2^19 rows and more, no shape (cwy_shape), or monitors that do not fit beside
// it.
static CwyPlan cwy_plan(int64_t n, int nl, int max_row, int monitors, size_t min_smem) {
  CwyPlan p;
  if (nl > kCwyMaxNl || max_row > 64 || n >= ((int64_t)1 << 19) || n < 1) return p;
  static_cast<CwyShape&>(p) = cwy_shape(n, sm_count() - monitors);
  if (p.G == 0) return CwyPlan();
  p.vs = cwy_smem_bytes(nl, p.chunk, p.rt, true) <= kCwySmemMax;
  p.smem = std::max(cwy_smem_bytes(nl, p.chunk, p.rt, p.vs), min_smem);
  const void* kern = p.vs ? (const void*)k_ar_cwy<true> : (const void*)k_ar_cwy<false>;
  int per = 0;
  if (p.smem > kCwySmemMax ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCwySmemMax) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, p.threads, p.smem) != cudaSuccess ||
      per * sm_count() < p.G + monitors) {
    (void)cudaGetLastError();
    return CwyPlan();
  }
  return p;
}
