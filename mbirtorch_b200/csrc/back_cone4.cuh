// Cone back projection at psf radius 1 for detectors of a multiple of four
// rows: the warp-per-cylinder scheme of back_cone_kernel with vector columns
// and two slices per instruction.
//
// A warp owns a pixel's chunk of 64 NP slices; lane l owns the slices l + 32
// i, two of them as the halves of one register pair (f2).  Per 32 views, each
// lane forms one view's record -- taps, vertical map, the rows that the chunk
// reaches and the form that its slices take -- into the warp's table, so that
// a view costs the warp three 16-byte broadcasts.  The view's detector column
// h(m) = sum_tc w_c sino[v, c + tc, m] is then formed four rows a lane (one
// 16-byte load per tap, with up to three such groups in flight), and each
// slice takes its three vertical taps from it.
//
// The vertical taps.  Slice k covers [m_p - w_r / 2, m_p + w_r / 2] with m_p =
// m0 + w_r k.  With mc = rint(m_p) and d = m_p - mc its overlaps with the rows
// either side of mc are
//     am = sat((w_r - 1) / 2 - d),   ap = sat((w_r - 1) / 2 + d)
// and with mc what is left, w_r - am - ap: the trapezoid weights of
// cone_beam.py:268-299 while w_r <= 2, where no slice reaches further rows
// and am, ap <= min(w_r, 1).  Taller slices (pixels nearer the source than
// the psf radius was chosen for) take the clamped trapezoid.
//
// What bounds it: the latency of the column loads (they come from L2: 20% of
// its rate) and the L1 data path (0.86 of its wavefronts); issue slots are
// 0.59 used.  back_cone_kernel was bound by issue: a headline subset step's
// gradient (1602 pixels x 256 slices x 720 views, 320 rows) took 605 M warp
// instructions, this form 301 M.  Measured, CUDA events: that gradient 643 ->
// 468 us, at 256^3 and 360 views 98.6 -> 77.5 us; whole volumes 77.6 -> 52.2 ms
// (headline), 1186 -> 650 us (128^3, 256 views).  Four CTAs per SM (64
// registers, a few spilled) against three without: 543 -> 468 us.  Not kept:
// prefetching the next view's columns to L1 (468 -> 538 us), leaving out the
// channel taps of zero weight (468 -> 465 us there, but 650 -> 700 us for the
// 128^3 volume), skipping the slice pairs past the band at run time (468 -> 488
// us; NP is picked to leave few).
#pragma once

#include "projectors.cuh"

namespace mbir {

constexpr int kBack4Pad = 24;  // zero rows either side of the column buffer

// What a slice chunk does at a view.
enum { kBackSkip = 0, kBackInside = 1, kBackClamped = 2, kBackGeneral = 3 };

struct __align__(16) Back4Rec {
  float w0, w1, w2, w_r;  // channel taps times the view's scale; rows per slice
  float m0, c1, a0, a1;   // m_p = m0 + w_r k; (w_r - 1) / 2; t(k) = a0 + a1 k
  int r0, r1, r2;         // the taps' sinogram columns v * C + c
  unsigned rows;          // first row / 4, last row << 12, form << 24
};

inline size_t back4_smem(int R) {
  return (size_t)(kThreads / 32) *
         (32 * sizeof(Back4Rec) + sizeof(float) * (R + 2 * kBack4Pad));
}

// Four rows' weighted taps of one column group into the column buffer.
template <int N, typename RD>
__device__ __forceinline__ void back4_columns(const RD &rd, const Back4Rec &r, int R, int m,
                                              int m_hi, unsigned h_s) {
  f2 a[N][3], b[N][3];
  const int c[3] = {r.r0, r.r1, r.r2};
#pragma unroll
  for (int u = 0; u < N; ++u) {
    // (the last group: lanes past the chunk's rows repeat its last row group)
    const int mu = u == N - 1 ? min(m + 128 * u, m_hi & ~3) : m + 128 * u;
#pragma unroll
    for (int t = 0; t < 3; ++t) rd.get4p((size_t)c[t] * R + mu, a[u][t], b[u][t]);
  }
  const f2 w0 = f2_dup(r.w0), w1 = f2_dup(r.w1), w2 = f2_dup(r.w2);
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const int mu = u == N - 1 ? min(m + 128 * u, m_hi & ~3) : m + 128 * u;
    const f2 x = f2_fma(w2, a[u][2], f2_fma(w1, a[u][1], f2_mul(w0, a[u][0])));
    const f2 y = f2_fma(w2, b[u][2], f2_fma(w1, b[u][1], f2_mul(w0, b[u][0])));
    sts_f2x2(h_s + 4u * (unsigned)mu, x, y);
  }
}

// The vertical taps of the lane's slice pairs kp.  CLAMP: slices may lie
// outside the column buffer's padding.
template <int CP, int NP, bool CLAMP>
__device__ __forceinline__ void back4_slices(f2 (&acc)[NP], const f2 (&kp)[NP],
                                             const Back4Rec &r, unsigned h_s, float lo, float hi) {
  const f2 m0 = f2_dup(r.m0), wr = f2_dup(r.w_r), a0 = f2_dup(r.a0), a1 = f2_dup(r.a1),
           one = f2_dup(1.f), magic = f2_dup(kRintMagic);
  const unsigned hm = h_s - 4u * kRintBits;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    f2 mp = f2_fma(wr, kp[j], m0);
    if (CLAMP) {
      float x, y;
      f2_unpack(mp, x, y);
      mp = f2_pack(fminf(fmaxf(x, lo), hi), fminf(fmaxf(y, lo), hi));
    }
    const f2 kr = f2_add(mp, magic);  // low bits: rint(m_p)
    float da, db, ka, kb;
    f2_unpack(f2_sub(mp, f2_sub(kr, magic)), da, db);
    f2_unpack(kr, ka, kb);
    f2 am = f2_pack(__saturatef(r.c1 - da), __saturatef(r.c1 - db));
    f2 ap = f2_pack(__saturatef(r.c1 + da), __saturatef(r.c1 + db));
    f2 ac = f2_sub(f2_sub(wr, am), ap);
    if (CP == 2) {
      am = f2_mul(am, am);
      ac = f2_mul(ac, ac);
      ap = f2_mul(ap, ap);
    }
    const unsigned sa = hm + 4u * __float_as_uint(ka), sb = hm + 4u * __float_as_uint(kb);
    const f2 xm = f2_pack(lds_f32(sa - 4u), lds_f32(sb - 4u));
    const f2 xc = f2_pack(lds_f32(sa), lds_f32(sb));
    const f2 xp = f2_pack(lds_f32(sa + 4u), lds_f32(sb + 4u));
    const f2 s = f2_fma(ap, xp, f2_fma(ac, xc, f2_mul(am, xm)));
    const f2 t = f2_fma(a1, kp[j], a0);
    const f2 q = f2_fma(t, t, one);
    f2 ic = q;  // coefficient power 2: 1 / cos^2 = 1 + t^2
    if (CP == 1) {
      float qa, qb;
      f2_unpack(q, qa, qb);
      ic = f2_mul(q, f2_pack(rsqrt_ftz(qa), rsqrt_ftz(qb)));
    }
    acc[j] = f2_fma(ic, s, acc[j]);
  }
}

template <int CP, int NP, typename RD>
__device__ __forceinline__ void back_cone4_kernel_body(
    Geo g, const float *__restrict__ vp, int v_start, int v_count, int vpc, RD rd,
    const int64_t *__restrict__ pix, int P, int slice_start, int band, int slice_chunks,
    float *__restrict__ out, const ConeFwdRec *__restrict__ recs) {
  MBIR_PDL_ENTRY();
  extern __shared__ float4 sm4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long gw = (long long)blockIdx.x * (kThreads / 32) + warp;
  const int p = (int)(gw / slice_chunks);
  if (p >= P) return;  // whole warp: no block-level barrier in this kernel
  const int sc = (int)(gw - (long long)p * slice_chunks);
  Back4Rec *tab = reinterpret_cast<Back4Rec *>(sm4) + warp * 32;
  float *h = reinterpret_cast<float *>(reinterpret_cast<Back4Rec *>(sm4) + kThreads) +
             warp * (g.R + 2 * kBack4Pad) + kBack4Pad;
  if (lane < kBack4Pad) h[lane - kBack4Pad] = h[g.R + lane] = 0.f;
  const unsigned h_s = (unsigned)__cvta_generic_to_shared(h);
  const int l0 = sc * 64 * NP, l_end = min(band, l0 + 64 * NP);
  const int chunk = blockIdx.y;
  const int vb = chunk * vpc, ve = min(v_count, vb + vpc);
  float xt, yt;
  pixel_xy(g, (int)pix[p], xt, yt);
  f2 acc[NP], kp[NP];  // (lanes past the band repeat its last slice)
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    acc[j] = 0;
    const int l = l0 + lane + 64 * j;
    kp[j] = f2_pack((float)(slice_start + min(l, band - 1)),
                    (float)(slice_start + min(l + 32, band - 1)));
  }
  const float kf = (float)(slice_start + l0), kl = (float)(slice_start + max(l_end - 1, l0));
  const float lo_clamp = -2.f, hi_clamp = (float)(g.R + 1);

  for (int vg = vb; vg < ve; vg += 32) {
    const int nv = min(32, ve - vg);
    __syncwarp();
    if (lane < nv) {
      Back4Rec r;
      float w[3];
      int ctr;
      if (CP == 1 && recs != nullptr) {
        // The same values cone_bin_kernel formed for this (view, slot).
        const ConeFwdRec fr = load_rec(recs + (size_t)(vg + lane) * P + p);
        ctr = __float_as_int(fr.c.z);
        w[0] = fr.b.y;
        w[1] = fr.b.z;
        w[2] = fr.b.w;
        r.m0 = fr.a.x;
        r.w_r = fr.a.y;
        r.a0 = fr.c.x;
        r.a1 = fr.c.y;
      } else {
        const int gv = v_start + vg + lane;
        const float ang = vp[2 * gv];
        const float z_off = __fsub_rn(g.rso, vp[2 * gv + 1]);
        const ConeVP q = cone_vp(g, ang, cosf(ang), sinf(ang), z_off, xt, yt);
        ctr = q.ctr;
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const float a = tap_weight(q.n_p, q.ctr + t - 1, q.half_w1, q.lmax, q.ws, g.C);
          w[t] = CP == 2 ? __fmul_rn(a, a) : a;
        }
        r.m0 = q.m0;
        r.w_r = q.w_r;
        cone_tcoef(g, q.mag, z_off, r.a0, r.a1);
      }
      const int v = vg + lane;
      const float scl = rd.scale(v);
      r.w0 = __fmul_rn(w[0], scl);
      r.w1 = __fmul_rn(w[1], scl);
      r.w2 = __fmul_rn(w[2], scl);
      r.c1 = 0.5f * (r.w_r - 1.f);
      r.r0 = v * g.C + min(max(ctr - 1, 0), g.C - 1);
      r.r1 = v * g.C + min(max(ctr, 0), g.C - 1);
      r.r2 = v * g.C + min(max(ctr + 1, 0), g.C - 1);
      // Rows this chunk's slices reach (the map is affine in k).
      const float ma = fmaf(r.w_r, kf, r.m0), mb = fmaf(r.w_r, kl, r.m0);
      const float mmin = fminf(ma, mb), mmax = fmaxf(ma, mb);
      const float lo = fmaxf(floorf(mmin) - 2.f, 0.f);
      const float hi = fminf(ceilf(mmax) + 2.f, (float)(g.R - 1));
      unsigned form = kBackSkip;
      unsigned rows = 0;
      if (lo <= hi) {
        const bool inside = mmin >= (float)(2 - kBack4Pad) && mmax <= (float)(g.R - 3 + kBack4Pad);
        form = r.w_r <= 2.f ? (inside ? kBackInside : kBackClamped) : kBackGeneral;
        rows = (unsigned)((int)lo >> 2) | ((unsigned)(int)hi << 12);
      }
      r.rows = rows | (form << 24);
      tab[lane] = r;
    }
    __syncwarp();
#pragma unroll 1
    for (int i = 0; i < nv; ++i) {
      const Back4Rec r = tab[i];
      const unsigned form = r.rows >> 24;
      if (form == kBackSkip) continue;  // uniform over the warp
      const int m_lo = (int)(r.rows & 0xfffu) * 4, m_hi = (int)((r.rows >> 12) & 0xfffu);
      int left = ((m_hi - m_lo) >> 7) + 1;  // groups of 128 rows
      int m = m_lo + 4 * lane;
      for (; left > 3; left -= 2, m += 256) back4_columns<2>(rd, r, g.R, m, m_hi, h_s);
      if (left == 3)
        back4_columns<3>(rd, r, g.R, m, m_hi, h_s);
      else if (left == 2)
        back4_columns<2>(rd, r, g.R, m, m_hi, h_s);
      else
        back4_columns<1>(rd, r, g.R, m, m_hi, h_s);
      __syncwarp();
      if (form == kBackInside) {
        back4_slices<CP, NP, false>(acc, kp, r, h_s, lo_clamp, hi_clamp);
      } else if (form == kBackClamped) {
        back4_slices<CP, NP, true>(acc, kp, r, h_s, lo_clamp, hi_clamp);
      } else {
        const float hw1r = 0.5f * (r.w_r + 1.f), lmaxr = fminf(r.w_r, 1.f);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          float k2[2], s2[2];
          f2_unpack(kp[j], k2[0], k2[1]);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float m_p = fminf(fmaxf(fmaf(r.w_r, k2[u], r.m0), lo_clamp), hi_clamp);
            const float mcf = rintf(m_p), d = m_p - mcf;
            const int mc = (int)mcf;
            float s = 0.f;
#pragma unroll
            for (int t = -1; t <= 1; ++t) {
              float a = trap_w<false>(hw1r - fabsf(d - (float)t), lmaxr);
              if (CP == 2) a = a * a;
              s = fmaf(a, h[mc + t], s);
            }
            const float tk = fmaf(r.a1, k2[u], r.a0);
            s2[u] = s * (CP == 2 ? fmaf(tk, tk, 1.f) : inv_cos_from_t(tk));
          }
          acc[j] = f2_add(acc[j], f2_pack(s2[0], s2[1]));
        }
      }
      __syncwarp();
    }
  }
  float *o = out + (size_t)chunk * P * band + (size_t)p * band;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const int l = l0 + lane + 64 * j;
    float a, b;
    f2_unpack(acc[j], a, b);
    if (l < band) o[l] = a;
    if (l + 32 < band) o[l + 32] = b;
  }
}

template <int CP, int NP, typename RD>
__global__ void __launch_bounds__(kThreads, NP == 1 ? 5 : 4)
back_cone4_kernel(Geo g, const float *__restrict__ vp, int v_start, int v_count, int vpc, RD rd,
                  const int64_t *__restrict__ pix, int P, int slice_start, int band,
                  int slice_chunks, float *__restrict__ out,
                  const ConeFwdRec *__restrict__ recs) {
  back_cone4_kernel_body<CP, NP, RD>(g, vp, v_start, v_count, vpc, rd, pix, P, slice_start, band,
                                     slice_chunks, out, recs);
}

}  // namespace mbir
