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
// O(L^2).  While |L| <= 1e-11 the correction L r is formed in FP32: its
// conversions, products and sums (19 roundings of 2^-25 on the way of an entry,
// at most 127 entries) are off by 6e-17 ||w|| at most, half of what the rounding
// of r is.  (In FP64 it costs 0.5 us a step: 100 x 100, istop 1, 308 -> 319 us.)
// Beyond, forward substitution in FP64.
//
// A block owns `chunk` rows of every vector.  With VS its rows of the whole
// basis stay in shared memory for the solve (n (nl - 1) <= ~3.5e6 on 152 SMs)
// and each pass reads them from there; otherwise the passes read the basis
// from L2.  A warp owns 32 rt of the block's rows and every kg-th vector, forms
// lane partials of the two dots in FP64 and sums them over the lanes and the
// grid on the integer pipe (fixsum.cuh).
//
// The window of V^T w: a lane partial is cut at 2^(ew-96) (unit vectors), so
// with at most 2^17 of them the coefficients are good to 2^-55 ||w|| while 2^ew
// is at most 2^24 ||w||.  ||w|| is known one reduction later, from h and beta:
// ||A|| places only the first step's window, and each step the next one's (12
// above).  A step whose window turns out wrong (vectors that do not meet the
// rows of the norm, scales far apart) is run once more, before anything of it
// is published, with the window from max |w| (an integer maximum over the grid
// and a barrier of its own).
#pragma once

struct CwyPlan : CwyShape {
  bool vs = false;
  size_t smem = 0;
};

constexpr int kCwyMaxNl = 128;
constexpr size_t kCwySmemMax = 220 * 1024;  // leaves the estimate monitors' static shared memory

// 64-bit words of one buffer of grid sums: r and l limbs per vector, then the
// four limbs of the norm, and at the offsets below from there the dots outside
// the window, the high word of max |w| and the norm's addends outside.
__host__ __device__ inline int cwy_acc_words(int nl) { return 4 * nl + 8; }
constexpr int kCwyBadDot = 4, kCwyMax = 5, kCwyBadNorm = 6;
constexpr int kCwyAbove = 24, kCwyNext = 12;  // of a window over log2 ||w||: at most, and for the next step
// ew and -il[k] (il: floor(log2 s_k), 1 / s_k = ||W_k||) from here up, so that a
// window's unit, at 2^(ew - il - 96) or 2^(1 - il - il - 96), is never far below
// the smallest double.
constexpr int kCwyMinExp = -489;
constexpr double kCwyLMax = 1e-11;  // largest |L| whose correction FP32 forms

static size_t cwy_smem_bytes(int nl, int chunk, int rt, bool vs) {
  const size_t nrg = (size_t)(chunk + 32 * rt - 1) / (32 * rt);
  size_t d = (size_t)chunk * (vs ? nl : 2) + 4 * (size_t)(nl + 2) + 4 * nrg * nl + 4 * 32;
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
  __shared__ int s_bad, s_slow, s_end, s_wrong, s_ew;
  __shared__ unsigned s_max[32];  // per warp
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
  long long* red4 = part + (size_t)4 * nrg * nl;      // [warp][4]
  float* rf = reinterpret_cast<float*>(red4 + 4 * 32);
  int* il = reinterpret_cast<int*>(rf + nl + 2);      // floor(log2 s_k), at most -kCwyMinExp
  float* Lf = reinterpret_cast<float*>(il + nl + 2);  // row k (0-based) of L at k (k - 1) / 2
  const int64_t r0 = (int64_t)b * chunk;
  const int nloc = (int)max((int64_t)0, min(r0 + chunk, st.n) - r0);
  const int aw = cwy_acc_words(nl);
  unsigned nb = 0;
  int last = 0;
  bool pending = false;   // beta of the step before is still to be formed
  bool measured = false;  // its window came from max |w|
  bool bad = false;       // a dot of it was outside the window
  bool measure = false;   // this step is run again
  int rr = 0;             // steps run, with the repeated ones: three buffers in turn
  const bool zero_x = c->done != 0;
  if (!zero_x) {
    const double* w1 = WAT(st, 1) + r0;
    for (int l = t; l < nloc; l += bd) Vs[l] = w1[l];
    if (t == 0) {
      ss[1] = st.s[1];
      il[1] = min(ilog2_normal(ss[1]), -kCwyMinExp);
      s_bad = s_slow = s_end = s_wrong = 0;
      s_ew = ew;
    }
    __syncthreads();
  }
  for (int i = 2; !zero_x; ++i) {
    const int nv = i - 1;
    // ---- w = scaling s_{i-1} A W_{i-1} on the block's rows (psfun_d_arnoldi.f90:202).
    // s_{i-1} is formed by one thread meanwhile (sqrt and division: ~1200 clocks).
    {
      const double* __restrict__ x = WAT(st, nv);
      for (int l = t; l < nloc && i <= nl; l += bd) {
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
      if (pending && t >= bd - 32) {  // the norm of the previous step (every block alike)
        const long long* pn = acc_all + (size_t)((rr + 2) % 3) * aw + 4 * nl;
        long long w4[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w4[q] = ld_relaxed_s64(pn + q);
        const bool badn = ld_relaxed_s64(pn + kCwyBadNorm) != 0;
        unsigned m = 0u;  // the high word of max |h| orders as the magnitude does
        for (int k = lane; k < nv - 1; k += 32) m = max(m, (unsigned)__double2hiint(hv[k]) & 0x7fffffffu);
        m = __reduce_max_sync(0xffffffffu, m);
        if (lead) {
          const double beta = badn ? __longlong_as_double(0x7ff8000000000000ll)
                                   : sqrt(scale_pow2(fix_units(w4), 2 * ew + 8 - 192));
          const int e = (int)(max(m, (unsigned)__double2hiint(beta) & 0x7fffffffu) >> 20) - 1023;  // of ||w||
          s_wrong = !measured && (bad || badn || ew > max(e + kCwyAbove, kCwyMinExp));
          if (!s_wrong) {
            s_ew = e > -1023 ? max(e + kCwyNext, kCwyMinExp) : ew;
            const double s = 1.0 / beta;
            if (i <= nl) {
              ss[nv] = s;
              il[nv] = min(ilog2_normal(s), -kCwyMinExp);
            }
            if (beta == 0.0 && i <= nl) s_end = 1;
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
        }
      }
      __syncthreads();
      const bool wrong = pending && s_wrong;
      pending = false;
      if (wrong) {  // the previous step again
        if (!VS) {  // its newest vector: this thread's rows
          for (int l = t; l < nloc; l += bd) Vs[l] = __ldcg(WAT(st, nv - 1) + r0 + l);
        }
        i -= 2;
        measure = true;
        continue;
      }
      if (i > nl) break;
      if (s_end) {  // h(i-1,i-2) == 0: the solve ends on the invariant subspace
        if (b == 0 && t == 0) c->done = 1;
        break;
      }
      ew = s_ew;
      const double f = scaling * ss[nv];
      for (int l = t; l < nloc; l += bd) wl[l] *= f;
      __syncthreads();
    }
    long long* acc = acc_all + (size_t)(rr % 3) * aw;
    const double* vl = VS ? Vs + (size_t)(nv - 1) * chunk : Vs;  // rows of W_{i-1}
    if (measure) {
      unsigned m = 0u;
      for (int l = t; l < nloc; l += bd) m = max(m, (unsigned)__double2hiint(wl[l]) & 0x7fffffffu);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) s_max[warp] = m;
      __syncthreads();
      if (warp == 0) {
        m = __reduce_max_sync(0xffffffffu, lane < (bd >> 5) ? s_max[lane] : 0u);
        if (lane == 0) atomicMax(reinterpret_cast<unsigned*>(acc + 4 * nl + kCwyMax), m);
      }
      if (!grid_sync_to(&c->bar_count, (++nb) * (unsigned)G, &c->err)) break;
      m = (unsigned)ld_relaxed_s64(acc + 4 * nl + kCwyMax);
      // ||w|| < 2^ew by sqrt(n) and two bits; w of zeros, and one that is not finite, keep what there is
      if (m > 0u && m < 0x7ff00000u)
        ew = max((int)(m >> 20) - 1021 + (33 - __clz((unsigned)max((int64_t)1, st.n - 1))) / 2, kCwyMinExp);
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
      if (t < 2 * nv - 1) {
        const int k = t < nv ? t : t - nv, sel = t < nv ? 0 : 2;
        long long h = 0, l = 0;
        for (int g = 0; g < nrg; ++g) {
          const long long* o = part + ((size_t)g * nl + k) * 4 + sel;
          h += o[0];
          l += o[1];
        }
        fix96_carry(h, l);
        long long* o = acc + (t < nv ? 0 : 2 * nl) + 2 * k;
        red_add_s64(o, h);
        red_add_s64(o + 1, l);
      }
      if (t == bd - 1) {
        if (s_bad) red_add_s64(acc + 4 * nl + kCwyBadDot, 1);
        s_bad = 0;
      }
    }
    if (!grid_sync_to(&c->bar_count, (++nb) * (unsigned)G, &c->err)) break;
    // all words of the step are fetched at once
    const bool stop = *(volatile int*)&c->stop_dec != 0;
    const long long bad_word = ld_relaxed_s64(acc + 4 * nl + kCwyBadDot);
    long long hi = 0, lo = 0;  // thread t < nv: r of vector t + 1; then l of vector t - nv + 1
    if (t < 2 * nv - 1) {
      const long long* o = acc + (t < nv ? 2 * t : 2 * nl + 2 * (t - nv));
      hi = ld_relaxed_s64(o);
      lo = ld_relaxed_s64(o + 1);
    }
    if (stop) {
      if (b == 0 && t == 0) c->done = 1;
      break;
    }
    bad = bad_word != 0;
    // ---- h = (I + L)^{-1} r
    if (t < 2 * nv - 1) {
      const bool isr = t < nv;
      const int k = isr ? t : t - nv;
      // times s_k (s_k s_{i-1}), their exponents taken into the window's
      double v = fix96_value(hi, lo, isr ? ew : 1) * scale_pow2(ss[k + 1], -il[k + 1]);
      if (!isr) v *= scale_pow2(ss[nv], -il[nv]);
      if (bad) v = __longlong_as_double(0x7ff8000000000000ll);
      if (isr) {
        rv[k] = v;
        rf[k] = (float)scale_pow2(v, -ew);  // |r_k| <= ||w||
      } else {
        lv[k] = v;
        Lf[(size_t)(nv - 1) * (nv - 2) / 2 + k] = (float)v;
        if (b == 0) Lg[(size_t)(nv - 1) * nl + k] = v;
        if (!(fabs(v) <= kCwyLMax) && (!bad || measure)) s_slow = 1;  // (a step that will be run again says nothing)
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
      for (int l = t; l < aw; l += bd) acc_all[(size_t)((rr + 1) % 3) * aw + l] = 0;
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
      long long w4[4];
      if (!fix192_limbs(p, 2 * ew + 8, w4)) s_bad = 1;
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // 24 bits at a time: 32 lanes of them fit an int
        const unsigned l = __reduce_add_sync(0xffffffffu, (unsigned)w4[q] & 0xffffffu);
        const unsigned h = __reduce_add_sync(0xffffffffu, (unsigned)(w4[q] >> 24));
        if (lane == 0) red4[warp * 4 + q] = (long long)l + ((long long)h << 24);
      }
      __syncthreads();
      if (t < 4) {  // a limb each, its carry into the next one's word
        long long q = 0, h = 0;
#pragma unroll 4
        for (int g = 0; g < (bd >> 5); ++g) q += red4[4 * g + t];
        if (t < 3) fix96_carry(h, q);
        red_add_s64(acc + 4 * nl + t, q);
        if (t < 3) red_add_s64(acc + 4 * nl + t + 1, h);
        if (t == 3 && s_bad) red_add_s64(acc + 4 * nl + kCwyBadNorm, 1);
        if (t == 3) s_bad = 0;
      }
    }
    if (!grid_sync_to(&c->bar_count, (++nb) * (unsigned)G, &c->err)) break;
    ++rr;
    pending = true;
    measured = measure;
    measure = false;
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
