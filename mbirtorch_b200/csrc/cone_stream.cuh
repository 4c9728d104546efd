// Cone forward projection over the channel-sorted bins, streamed by channel.
//
// One CTA owns (view, `bpc` blocks of kFwdCB channels, one or two) and walks
// its run of the sorted list.  Lane l of warp w owns the detector rows 64 w + l and
// 64 w + l + 32, as the halves of register pairs (f2), so that the work that
// a warp does once per pixel is shared by 64 rows and most arithmetic is one
// instruction for both rows.
//
// The pixels come in nondecreasing centre channel, so only three channel
// sums are open at a time.  They stay in registers, and when the centre moves
// on, the channel that no later pixel reaches goes straight to the epilogue
// (which has had its operands in flight for two channels).  No accumulator
// in shared memory, no pass over it at the end, and a CTA's channel run may
// be as long as the grid allows.
//
// The vertical footprint.  A pixel's slices tile the detector column: slice k
// covers m0 + w_r (k -+ 1/2), and row m collects the overlap of each slice
// with [m - 1/2, m + 1/2] (the trapezoid weight of cone_beam.py:203-226).
// With k_m = (m - m0) / w_r the row's centre in slices, kc = rint(k_m) and
// d = w_r (kc - k_m), the neighbours of slice kc overlap the row by
//     kc - 1: am = sat((1 - w_r) / 2 + d),   kc + 1: ap = sat((1 - w_r) / 2 - d)
// and slice kc by what is left, 1 - am - ap: the same three weights as the
// trapezoid's while w_r >= 1/2, where |d| <= w_r / 2 keeps am and ap at or
// below 1/2 <= min(w_r, 1), so that no upper clamp acts and no further slice
// reaches the row.  Pixels with flatter slices take the general form, one
// pixel at a time.
//
// What bounds it: issue slots (0.67-0.72 of them used; no pipe and no memory
// level is above 0.59).  One row per thread with the sums in shared memory
// (forward_cone_binned_kernel) took 1028 M warp instructions for a headline
// subset step (1602 pixels x 256 slices x 720 views, 320 x 768 detector), this
// form 722 M; half of them are the walk, a quarter the epilogue's stores
// and line-search sums.  Measured, CUDA events: that step's forward 1194 ->
// 896 us; whole volumes 108.8 -> 78.5 ms (headline), 12.2 -> 8.4 ms (256^3,
// 360 views), 1178 -> 964 us (128^3, 256 views).  Not kept: padding wide
// enough to leave out the clamps (its shared memory cost CTAs: 64-row
// detectors 105 -> 178 us), 64-register code for one- and two-warp CTAs (99
// -> 106 us).
#pragma once

#include <type_traits>

#include "projectors.cuh"

namespace mbir {

constexpr int kStreamCap = 64;     // records per round
constexpr int kStreamRows = 64;    // detector rows per warp
constexpr int kStreamPad = 4;      // zeros either side of a staged cylinder

// A record in shared memory: the walk's operands as pairs of equal halves.
struct __align__(16) StreamRec {
  float inv[2], nm[2];   // k_m = m * inv + nm, inv = 1 / w_r
  float w_r;
  int slot;              // centre channel - c0
  float w2[2];           // channel tap at centre + 1
  float w0[2], w1[2];    // channel taps at centre - 1 and centre
  float t0, t1;          // tangent of the ray's slope at slice k: t0 + t1 k
  int row, unused;       // row of `values`
};

__host__ __device__ inline int stream_pitch(int band) {
  return ((band + 3) & ~3) + 2 * kStreamPad;
}

__host__ __device__ inline size_t stream_smem(int band, int eb) {
  return sizeof(StreamRec) * kStreamCap + sizeof(float) * 2 * eb * stream_pitch(band);
}

__device__ __forceinline__ void cp_async16_s(unsigned dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4_s(unsigned dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}

// VEC: cylinders of a multiple of 4 slices from a 16-byte aligned array,
// copied and scaled four slices at a time; else one at a time.  EB: pixels
// staged per batch (a multiple of 4, at most 32).
template <typename EPI, bool VEC, int EB>
__device__ __forceinline__ void forward_cone_stream_kernel_body(
    Geo g, int v_start, const float *__restrict__ values, int P, int band,
    const ConeFwdRec *__restrict__ recs, const int *__restrict__ list,
    const int *__restrict__ offs, unsigned char *__restrict__ touched, int nblk, int bpc,
    EPI epi) {
  MBIR_PDL_ENTRY();
  extern __shared__ float4 sm4[];
  const int nthr = blockDim.x, tid = threadIdx.x, lane = tid & 31;
  constexpr int pad = kStreamPad;
  const int SP = stream_pitch(band);
  StreamRec *rec = reinterpret_cast<StreamRec *>(sm4);
  float *stage = reinterpret_cast<float *>(rec + kStreamCap);
  const bool vf = EPI::kViewFastest;
  const int grp = vf ? blockIdx.y : blockIdx.x, vl = vf ? blockIdx.x : blockIdx.y;
  const int f0 = grp * bpc;  // the CTA's first block
  int c0 = f0 * kFwdCB;
  int nch = min(bpc * kFwdCB, g.C - c0);
  const int nkeys = fwd_nkeys(g.C);
  const ConeFwdRec *vrec = recs + (size_t)vl * P;
  const int *vlist = list + (size_t)vl * P;
  const int *voffs = offs + (size_t)vl * (nkeys + 1);
  int start = voffs[c0], end = voffs[min(c0 + nch + 2, nkeys)];
  const int v = v_start + vl;
  if constexpr (!EPI::kViewFastest) {
    // Of two blocks, one that no pixel reaches is no part of the step: its
    // cells, which may be dead, are neither read nor counted.
    if (nch > kFwdCB) {
      const int second = voffs[c0 + kFwdCB], first_end = voffs[c0 + kFwdCB + 2];
      if (first_end == start) {
        start = second;
        c0 += kFwdCB;
        nch -= kFwdCB;
      } else if (second == end) {
        end = first_end;
        nch = kFwdCB;
      }
    }
  }
  for (int b = f0 + tid; b < min(f0 + bpc, nblk); b += nthr)
    touched[(size_t)v * nblk + b] =
        end > start && b * kFwdCB >= c0 && b * kFwdCB < c0 + nch;
  if (end == start) {
    epi.empty_tile(v, c0, nch);
    epi.begin(v);
    epi.end(v * nblk + f0);
    EPI::Stream::pad_partials(epi, v * nblk + f0 + 1, v * nblk + min(f0 + bpc, nblk));
    return;
  }
  // Zeros either side of each staged cylinder (the interiors are written by
  // every batch before they are read).
  const int pads = SP - band;  // pad before, and pad and the band's round-up behind
  for (int e = tid >> 5; e < 2 * EB; e += nthr >> 5)
    for (int o = lane; o < pads; o += 32) stage[e * SP + (o < pad ? o : band + o)] = 0.f;
  const int wr0 = (tid >> 5) * kStreamRows;
  const int m0 = wr0 + lane, m1 = m0 + kStreamStep;
  const int wr1 = min(wr0 + kStreamRows, g.R) - 1;  // the warp's last row
  const float mf0 = (float)min(m0, g.R - 1), mf1 = (float)min(m1, g.R - 1);
  const f2 mf = f2_pack(mf0, mf1);
  const float kc_lo = -2.f, kc_hi = (float)(band + 1);
  typename EPI::Stream stream(epi, v, c0, nch, m0);

  // The open channel sums: centre slot cj - 1, cj, cj + 1 (slot s is channel
  // c0 + s).  The centre slots of the list are -1 .. nch.
  int cj = -1;
  f2 q0 = 0, q1 = 0, q2 = 0;
  auto advance = [&](int to) {
#pragma unroll 1
    while (cj < to) {
      stream.put(cj - 1, q0);
      q0 = q1;
      q1 = q2;
      q2 = 0;
      ++cj;
    }
  };

  auto add = [&](int j, f2 w0, f2 w1, f2 w2, f2 det) {
    if (j != cj) advance(j);  // uniform over the warp; j > cj
    q0 = f2_fma(w0, det, q0);
    q1 = f2_fma(w1, det, q1);
    q2 = f2_fma(w2, det, q2);
  };

  // Staging: teams of 2^tw threads take the batch's pixels in turn, each
  // thread every 2^tw-th 16-byte (or 4-byte) chunk of the cylinder.  The
  // thread that copies a chunk also scales it, so the copy needs no barrier
  // of its own.
  constexpr int W = VEC ? 4 : 1;
  const int nq = band / W;
  const int tw = nq >= 32 ? 5 : 32 - __clz(nq - 1);  // (nq = 1: 0)
  const int T = 1 << tw, team = tid >> tw, tl = tid & (T - 1), teams = nthr >> tw;
  const unsigned SP4 = 4u * (unsigned)SP;
  const float *values_tl = values + W * tl;
  // slices 4 tl .. 4 tl + 3 as floats, and the step to the team's next chunk
  const float k0 = (float)(4 * tl);
  const f2 kfa = f2_pack(k0, k0 + 1.f), kfb = f2_pack(k0 + 2.f, k0 + 3.f),
           kstep = f2_dup((float)(4 * T));
  const unsigned rec_s0 = (unsigned)__cvta_generic_to_shared(rec);
  const unsigned st_s0 = (unsigned)__cvta_generic_to_shared(stage) + 4u * pad;
  const unsigned mine_s = st_s0 + 4u * W * tl + team * SP4;  // the first chunk copied here
  const f2 magic = f2_dup(kRintMagic), one = f2_dup(1.f);

  for (int base = start; base < end; base += kStreamCap) {
    const int n = min(kStreamCap, end - base);
    __syncthreads();  // the last round's records and buffers are free
    for (int i = tid; i < n; i += nthr) {
      const ConeFwdRec r = vrec[vlist[base + i]];
      StreamRec s;
      const float inv = r.b.x, nm = -r.a.x * inv;
      s.inv[0] = s.inv[1] = inv;
      s.nm[0] = s.nm[1] = nm;
      s.w0[0] = s.w0[1] = r.b.y;
      s.w1[0] = s.w1[1] = r.b.z;
      s.w2[0] = s.w2[1] = r.b.w;
      s.w_r = r.a.y;
      s.t0 = r.c.x;
      s.t1 = r.c.y;
      s.row = __float_as_int(r.c.w);
      s.slot = __float_as_int(r.c.z) - c0;
      rec[i] = s;
    }
    __syncthreads();
    const int nbat = (n + EB - 1) / EB;
    // Copies batch b (this thread's chunks).
    auto issue = [&](int b) {
      const int e0 = b * EB, nb = min(EB, n - e0);
      unsigned dst = mine_s + (b & 1) * EB * SP4;
      unsigned ra = rec_s0 + (unsigned)(e0 + team) * (unsigned)sizeof(StreamRec);
#pragma unroll 1
      for (int e = team; e < nb; e += teams) {
        const float *src = values_tl + (size_t)lds_u32(ra + 56u) * band;
        unsigned d = dst;
#pragma unroll 2
        for (int q = tl; q < nq; q += T) {
          if constexpr (VEC)
            cp_async16_s(d, src);
          else
            cp_async4_s(d, src);
          d += 4u * W * T;
          src += W * T;
        }
        dst += teams * SP4;
        ra += teams * (unsigned)sizeof(StreamRec);
      }
      cp_async_commit();
    };
    issue(0);
    for (int b = 0; b < nbat; ++b) {
      const int e0 = b * EB, nb = min(EB, n - e0);
      const unsigned rec_s = rec_s0 + (unsigned)e0 * (unsigned)sizeof(StreamRec);
      const unsigned buf_s = (b & 1) * EB * SP4;
      cp_async_wait<0>();  // this thread's chunks of batch b have landed
      unsigned p = mine_s + buf_s, ra = rec_s + team * (unsigned)sizeof(StreamRec);
#pragma unroll 1
      for (int e = team; e < nb; e += teams) {
        float t0, t1;
        lds_f32x2(ra + 48u, t0, t1);
        unsigned d = p;
        if constexpr (VEC) {
          const f2 t1d = f2_dup(t1), t0d = f2_dup(t0);
          f2 ka = kfa, kb = kfb;
#pragma unroll 2
          for (int q = tl; q < nq; q += T) {
            f2 xa, xb;
            lds_f2x2(d, xa, xb);
            const f2 ta = f2_fma(t1d, ka, t0d), tb = f2_fma(t1d, kb, t0d);
            const f2 qa = f2_fma(ta, ta, one), qb = f2_fma(tb, tb, one);
            float c0_, c1_, c2_, c3_;
            f2_unpack(qa, c0_, c1_);
            f2_unpack(qb, c2_, c3_);
            xa = f2_mul(xa, f2_mul(qa, f2_pack(rsqrt_ftz(c0_), rsqrt_ftz(c1_))));
            xb = f2_mul(xb, f2_mul(qb, f2_pack(rsqrt_ftz(c2_), rsqrt_ftz(c3_))));
            sts_f2x2(d, xa, xb);
            d += 16u * T;
            ka = f2_add(ka, kstep);
            kb = f2_add(kb, kstep);
          }
        } else {
          float k = (float)tl;
          for (int q = tl; q < nq; q += T) {
            sts_f32(d, lds_f32(d) * inv_cos_from_t_ftz(fmaf(t1, k, t0)));
            d += 4u * T;
            k += (float)T;
          }
        }
        p += teams * SP4;
        ra += teams * (unsigned)sizeof(StreamRec);
      }
      __syncthreads();  // batch b is staged; the other buffer's walkers are done
      if (b + 1 < nbat) issue(b + 1);

      // The pixels that the warp walks: a row meets the band only when its
      // centre slice lies in [-2, band + 1], so the warp skips a pixel whose
      // slices map all its rows, widened by one either side, outside.
      // `fast`: the three-weight form holds.
      unsigned todo, fast;
      {
        bool on = false, fs = false;
        if (lane < nb) {
          const unsigned r = rec_s + (unsigned)lane * (unsigned)sizeof(StreamRec);
          const float inv = lds_f32(r), nm = lds_f32(r + 8u);
          on = !(fmaf((float)(wr1 + 1), inv, nm) < kc_lo ||
                 fmaf((float)(wr0 - 1), inv, nm) > kc_hi);
          fs = lds_f32(r + 16u) >= 0.5f;
        }
        todo = __ballot_sync(0xffffffffu, on);
        fast = __ballot_sync(0xffffffffu, fs);
      }
      const unsigned st_s = st_s0 + buf_s - 4u * kRintBits;
      // The sums of N pixels over their slices for the lane's two rows, and
      // their channel taps, added in list order.  The loads of all N are in
      // flight together.
      auto walk = [&](auto count, const int (&e)[4]) {
        constexpr int N = decltype(count)::value;
        f2 km[N], wj[N], w2[N], fr[N], kr[N], det[N];
        unsigned ra[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
          f2 inv, nm;
          ra[u] = rec_s + (unsigned)e[u] * (unsigned)sizeof(StreamRec);
          lds_f2x2(ra[u], inv, nm);
          lds_f2x2(ra[u] + 16u, wj[u], w2[u]);
          // (clamped: a row whose centre slice lies outside meets zeros only)
          float ka, kb;
          f2_unpack(f2_fma(mf, inv, nm), ka, kb);
          km[u] = f2_pack(fminf(fmaxf(ka, kc_lo), kc_hi), fminf(fmaxf(kb, kc_lo), kc_hi));
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
          kr[u] = f2_add(km[u], magic);  // low bits: rint(k_m)
          fr[u] = f2_sub(f2_sub(kr[u], magic), km[u]);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
          float ka, kb;
          f2_unpack(kr[u], ka, kb);
          const unsigned se = st_s + (unsigned)e[u] * SP4;
          const unsigned sa = se + 4u * __float_as_uint(ka), sb = se + 4u * __float_as_uint(kb);
          const f2 xm = f2_pack(lds_f32(sa - 4u), lds_f32(sb - 4u));
          const f2 x0 = f2_pack(lds_f32(sa), lds_f32(sb));
          const f2 xp = f2_pack(lds_f32(sa + 4u), lds_f32(sb + 4u));
          float fa, fb, w_r, jf;
          f2_unpack(fr[u], fa, fb);
          f2_unpack(wj[u], w_r, jf);
          const float c1 = fmaf(-0.5f, w_r, 0.5f);
          const f2 am = f2_pack(__saturatef(fmaf(fa, w_r, c1)), __saturatef(fmaf(fb, w_r, c1)));
          const f2 ap = f2_pack(__saturatef(fmaf(-fa, w_r, c1)), __saturatef(fmaf(-fb, w_r, c1)));
          const f2 a0 = f2_sub(f2_sub(one, am), ap);
          det[u] = f2_fma(ap, xp, f2_fma(a0, x0, f2_mul(am, xm)));
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
          f2 w0, w1;
          float w_r, jf;
          lds_f2x2(ra[u] + 32u, w0, w1);
          f2_unpack(wj[u], w_r, jf);
          add(__float_as_int(jf), w0, w1, w2[u], det[u]);
        }
      };
      bool crowded = false;
      if constexpr (!EPI::kViewFastest) {
        if (nch > kFwdCB)
          crowded = stream.crowded(
              (int)lds_u32(rec_s + (unsigned)(nb - 1) * (unsigned)sizeof(StreamRec) + 20u) - cj);
      }
#pragma unroll 1
      for (int e4 = 0; e4 < nb; e4 += 4) {
        if constexpr (!EPI::kViewFastest) {
          if (crowded) stream.add_up();
        }
        unsigned four = (todo >> e4) & 15u;
        if (four == 15u && ((fast >> e4) & 15u) == 15u) {  // uniform over the warp
          walk(std::integral_constant<int, 4>{}, {e4, e4 + 1, e4 + 2, e4 + 3});
          continue;
        }
#pragma unroll 1
        while (four) {
          const int e = e4 + __ffs(four) - 1;
          four &= four - 1u;
          if ((fast >> e) & 1u) {
            walk(std::integral_constant<int, 1>{}, {e, 0, 0, 0});
            continue;
          }
          // The taps around each row's centre slice, clamped to the padding.
          const StreamRec &r = rec[e0 + e];
          const float *st = stage + ((b & 1) * EB + e) * SP + pad;
          const float w_r = r.w_r, hw1r = 0.5f * (w_r + 1.f), lmaxr = fminf(w_r, 1.f);
          float d2[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float k_m = fmaf(u ? mf1 : mf0, r.inv[0], r.nm[0]);
            const float kc = fminf(fmaxf(rintf(k_m), kc_lo), kc_hi);
            const float d = w_r * (kc - k_m);
            const int k = (int)kc;
            float s = 0.f;
#pragma unroll
            for (int ko = -1; ko <= 1; ++ko)
              s = fmaf(fminf(__saturatef(hw1r - fabsf(fmaf(w_r, (float)ko, d))), lmaxr), st[k + ko],
                       s);
            d2[u] = s;
          }
          add(r.slot, f2_dup(r.w0[0]), f2_dup(r.w1[0]), f2_dup(r.w2[0]), f2_pack(d2[0], d2[1]));
        }
      }
      stream.flush();
    }
  }
  advance(nch + 1);
  stream.finish(epi);
  epi.end(v * nblk + f0);
  EPI::Stream::pad_partials(epi, v * nblk + f0 + 1, v * nblk + min(f0 + bpc, nblk));
}

// WIDE: detectors of more than kStreamRows * 2 rows (three warps or more a
// CTA); else at most two warps a CTA, which have room for more registers.
template <typename EPI, bool VEC, int EB, bool WIDE>
__global__ void __launch_bounds__(WIDE ? 512 : 64, WIDE ? 2 : 12)
forward_cone_stream_kernel(Geo g, int v_start, const float *__restrict__ values, int P, int band,
                           const ConeFwdRec *__restrict__ recs, const int *__restrict__ list,
                           const int *__restrict__ offs, unsigned char *__restrict__ touched,
                           int nblk, int bpc, EPI epi) {
  forward_cone_stream_kernel_body<EPI, VEC, EB>(g, v_start, values, P, band, recs, list, offs,
                                                touched, nblk, bpc, epi);
}

}  // namespace mbir
