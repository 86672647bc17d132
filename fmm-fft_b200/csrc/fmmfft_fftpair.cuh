/*
 * FP32 FFT passes with two sequences a thread, sm_100a: the register Stockham pass k_fft_reg in packed
 * arithmetic (add, sub, mul, fma.rn.f32x2).
 *
 * Bound by instructions and shared-memory wavefronts before memory: a pass of length 512 takes 95
 * instructions a value in k_fft_reg, 50 here, and two exchanges whatever the orders of its input and
 * output (the threads' order changes between stages, not after them).  Measured (us, FP32): 2^26, P =
 * 256: combine 269 -> 209, passes 274 / 258 -> 240 / 201 (floor 164 each); 2^24, P = 64: combine 53 -> 47,
 * passes 76 / 70 -> 70 / 59 (floor 41); two blocks of 512 threads an SM still leave memory idle while
 * both compute.  Here a thread's registers hold the same element of two sequences, real parts in one
 * 64-bit pair and imaginary parts in another, so that every addition, twiddle and exchange (16-byte
 * accesses) serves both, a stage twiddle is read once for two values, and a multiplication by -i stays a
 * renaming.  Neighbouring sequences make a pair, so that an order across sequences has 16-byte global
 * accesses where the address allows.  Loads come before the twiddles are staged, as there.
 *
 * Exchange layout: 16-byte elements, element i of pair p at p * pitch + swz(i), swz(i) = i ^ (i / 8 mod
 * 8): a quarter-warp's 8 accesses (neighbouring elements, or stride 8, or neighbouring pairs, pitch
 * 8 / pairs mod 8) fall on 8 different 16-byte columns.  The swizzle is linear over XOR, so with a
 * constant length an address costs one XOR or none.
 */
#pragma once

struct Pair { /* a complex value of two sequences */
  float2 re, im;
};
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ Pair padd(Pair a, Pair b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Pair psub(Pair a, Pair b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
/* a w, both of two values; nwi = -w.im */
__device__ __forceinline__ Pair pmul(Pair a, float2 wr, float2 wi, float2 nwi) {
  return {ffma2(a.re, wr, mul2(a.im, nwi)), ffma2(a.re, wi, mul2(a.im, wr))};
}
__device__ __forceinline__ Pair pmul(Pair a, float2 w) { /* one twiddle for both */
  return pmul(a, make_float2(w.x, w.x), make_float2(w.y, w.y), make_float2(-w.y, -w.y));
}
__device__ __forceinline__ void pdft4(Pair &a, Pair &b, Pair &c, Pair &d) {
  const Pair t0 = padd(a, c), t1 = psub(a, c), t2 = padd(b, d), u = psub(b, d);
  a = padd(t0, t2), c = psub(t0, t2);
  b = {add2(t1.re, u.im), sub2(t1.im, u.re)}; /* t1 - i u */
  d = {sub2(t1.re, u.im), add2(t1.im, u.re)};
}
__device__ __forceinline__ void pdft8(Pair (&v)[8]) {
  const float2 h = make_float2(0.70710678118654752440f, 0.70710678118654752440f), nh = make_float2(-h.x, -h.x);
  pdft4(v[0], v[2], v[4], v[6]);
  pdft4(v[1], v[3], v[5], v[7]);
  /* o_k exp(-2 pi i k / 8) */
  const Pair o1 = {mul2(h, add2(v[3].re, v[3].im)), mul2(h, sub2(v[3].im, v[3].re))};
  const Pair s2 = v[5]; /* times -i: re = im, im = -re */
  const Pair o3 = {mul2(h, sub2(v[7].im, v[7].re)), mul2(nh, add2(v[7].re, v[7].im))};
  const Pair e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
  v[0] = padd(e0, o0), v[4] = psub(e0, o0);
  v[1] = padd(e1, o1), v[5] = psub(e1, o1);
  v[2] = {add2(e2.re, s2.im), sub2(e2.im, s2.re)}, v[6] = {sub2(e2.re, s2.im), add2(e2.im, s2.re)};
  v[3] = padd(e3, o3), v[7] = psub(e3, o3);
}

__host__ __device__ __forceinline__ int pair_pitch(int L, int np) { return L + (np >= 8 ? 1 : np == 1 ? 0 : 8 / np); }
__device__ __forceinline__ int pair_swz(int i) { return i ^ ((i >> 3) & 7); }
__device__ __forceinline__ int pair_at(int si, int c) { /* swz(i | c) from swz(i), no common bits */
  const int z = pair_swz(c);
  return (si ^ (z & 7)) + (z & ~7);
}
/* Shared bytes: exchange, stage twiddles, 4-step twiddle steps */
__host__ __device__ __forceinline__ size_t pair_smem(int L, int np) {
  return 16 * ((size_t)np * pair_pitch(L, np) + 9 * (size_t)np) + 8 * (size_t)L;
}
__device__ __forceinline__ float4 pair_pack(Pair v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }
__device__ __forceinline__ Pair pair_unpack(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }

/* The loaders' pair forms: sequences g and g + 1. */
struct StridedLd2 : StridedLd<float> {
  template <bool TIN> __device__ __forceinline__ void load(long row, unsigned g, int t, int q, Pair (&v)[8]) const {
    const float2 *const b = in + row * irow, *const sp = b + g * iseq + t * istr;
    const unsigned qs = (unsigned)q * istr;
    if (!TIN && iseq == 1 && ((uintptr_t)b & 15) == 0) { /* both in one 16-byte load (g and istr are even) */
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 a = *reinterpret_cast<const float4 *>(sp + r * qs);
        v[r] = {make_float2(a.x, a.z), make_float2(a.y, a.w)};
      }
    } else {
      const float2 *const sq = sp + iseq;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float2 a = sp[r * qs], c = sq[r * qs];
        v[r] = {make_float2(a.x, c.x), make_float2(a.y, c.y)};
      }
    }
  }
  __device__ __forceinline__ void finish(long, int, int, Pair (&)[8]) const {}
  /* a later block's input towards L2: W sequences of L values from g0 on */
  template <bool TIN> __device__ __forceinline__ void ahead(long row, unsigned g0, int W, int L) const {
    const float2 *const b = in + row * irow + g0 * iseq;
    if (TIN) {
      for (int e = threadIdx.x * 16; e < W * L; e += blockDim.x * 16)
        asm volatile("prefetch.global.L2 [%0];" : : "l"(b + (e / L) * iseq + (e & (L - 1))));
    } else {
      for (int e = threadIdx.x; e < L; e += blockDim.x) asm volatile("prefetch.global.L2 [%0];" : : "l"(b + e * (long)istr));
    }
  }
  static constexpr bool kAhead = true, kOwnOut = false;
};
struct CombineLd2 : CombineLd<float> { /* columns m, m + 1 (even m: 8-byte loads of the planar field) */
  static constexpr bool kAhead = false, kOwnOut = true; /* its output is the plan's own, 16-byte aligned */
  template <bool> __device__ __forceinline__ void load(long row, unsigned mc, int t, int q, Pair (&v)[8]) const {
    const long m = m0 + mc;
    const float *xt = this->xt + row * 2 * P * M, *u = this->u + row * 2 * (P - 1) * M;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int sc = t + r * q;
      const float *const p = (sc == 0 ? xt : u + (2L * (sc - 1)) * M) + m;
      v[r] = {*reinterpret_cast<const float2 *>(p), *reinterpret_cast<const float2 *>(p + M)};
    }
  }
  __device__ __forceinline__ void finish(long row, int t, int q, Pair (&v)[8]) const {
    const float2 *ssum = this->ssum + row * P;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int sc = t + r * q;
      if (sc == 0) continue;
      const float2 S = ssum[sc];
      const float sx = S.x * invM, sy = S.y * invM;
      v[r] = pmul({add2(v[r].re, make_float2(sy, sy)), sub2(v[r].im, make_float2(sx, sx))}, pretw[sc]);
    }
  }
};

/* Blocks of 512 threads, two an SM, also ask L2 for the input of the block that follows in their place
 * (2^24, P = 64: passes 72 / 63 us -> 70 / 59). */
constexpr unsigned kPairAhead = 2 * 148; /* a distance only: on another number of SMs a block asks too early or late */

/* L = 2^LGT (LGT = 0: any); q L / 8 threads a pair of sequences, W / 2 pairs a block.  TIN and TOUT as in
 * k_fft_reg. */
template <bool TIN, bool TOUT, class Ld, int LGT>
__global__ void __launch_bounds__(512, 2)
    k_fft_pair(const Ld ld, float2 *__restrict__ out, const float2 *__restrict__ twD, const float2 *__restrict__ twP, FftPass fp,
               const OutTab ot) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = LGT ? 1 << LGT : fp.L, np = fp.W >> 1, q = L >> 3;
  const int lg = LGT ? LGT : __ffs(L) - 1, lq = lg - 3, lnp = __ffs(np) - 1;
  const int LP = pair_pitch(L, np), tid = threadIdx.x;
  const unsigned g0 = blockIdx.x * (unsigned)fp.W;
  const long row = blockIdx.y;
  float4 *const buf = reinterpret_cast<float4 *>(smem_raw), *const twq = buf + np * LP;
  float2 *const twl = reinterpret_cast<float2 *>(twq + 9 * np); /* stage-major, as in k_fft_reg */
  int t, p;
  if (TIN) t = tid & (q - 1), p = tid >> lq;
  else p = tid & (np - 1), t = tid >> lnp;
  Pair v[8];
  ld.template load<TIN>(row, g0 + 2 * p, t, q, v);
  if constexpr (Ld::kAhead)
    if (blockDim.x == 512) {
      const unsigned nb = blockIdx.x + blockIdx.y * gridDim.x + kPairAhead, ny = nb / gridDim.x, nx = nb - ny * gridDim.x;
      if (ny < gridDim.y) ld.template ahead<TIN>(ny, nx * (unsigned)fp.W, fp.W, L);
    }
  auto post = [&](unsigned gi) -> float2 {
    const unsigned e = (gi * fp.twmul) & fp.twmask;
    if (fp.twbits == 0) return twP[e];
    const unsigned lo = (1u << fp.twbits) - 1;
    return cmul(twP[lo + 1 + (e >> fp.twbits)], twP[e & lo]);
  };
  const int ns0 = lg % 3 == 0 ? 8 : lg % 3 == 2 ? 4 : 2;
  for (int Ns = ns0; Ns <= q; Ns <<= 3)
    for (int m = tid; m < 7 * Ns; m += blockDim.x) {
      const int k = m / 7, r = m - 7 * k + 1;
      twl[Ns - ns0 + m] = twD[(long)(r * k * (q / Ns)) * fp.tws];
    }
  if (fp.twiddle_post)
    for (int m = tid; m < 8 * np; m += blockDim.x) {
      const unsigned g = g0 + 2 * (m >> 3), qr = (unsigned)q * (unsigned)(m & 7);
      const float2 a = post(g * qr), b = post((g + 1) * qr);
      twq[(m >> 3) * 9 + (m & 7)] = make_float4(a.x, b.x, a.y, b.y);
    }
  ld.finish(row, t, q, v);
  float4 *bw = buf + p * LP;
  int Ns, lNs;
  if (lg % 3 == 0) { /* radix 8: outputs 8t + r */
    pdft8(v);
    const int s0 = pair_swz(8 * t);
#pragma unroll
    for (int r = 0; r < 8; ++r) bw[pair_at(s0, r)] = pair_pack(v[r]);
    Ns = 8, lNs = 3;
  } else if (lg % 3 == 2) { /* radix 4: butterflies t and t + q */
    pdft4(v[0], v[2], v[4], v[6]);
    pdft4(v[1], v[3], v[5], v[7]);
    const int s0 = pair_swz(4 * t);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      bw[pair_at(s0, r)] = pair_pack(v[2 * r]);
      bw[pair_at(s0, 4 * q + r)] = pair_pack(v[2 * r + 1]);
    }
    Ns = 4, lNs = 2;
  } else { /* radix 2: butterflies t + m q */
    const int s0 = pair_swz(2 * t);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      bw[pair_at(s0, 2 * m * q)] = pair_pack(padd(v[m], v[m + 4]));
      bw[pair_at(s0, 2 * m * q + 1)] = pair_pack(psub(v[m], v[m + 4]));
    }
    Ns = 2, lNs = 1;
  }
  const int nst = (lg - lNs) / 3;
  /* any thread may take any butterfly of a later stage: from here on threads lie as the output wants them */
  if (TOUT != TIN) {
    if (TOUT) t = tid & (q - 1), p = tid >> lq;
    else p = tid & (np - 1), t = tid >> lnp;
    bw = buf + p * LP;
  }
  const int st = pair_swz(t);
#pragma unroll
  for (int si = 0; si < (LGT ? (LGT - (LGT % 3 == 0 ? 3 : LGT % 3)) / 3 : nst); ++si) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = pair_unpack(bw[pair_at(st, r * q)]);
    const int k = t & (Ns - 1), tb = Ns - ns0 + 7 * k - 1;
#pragma unroll
    for (int r = 1; r < 8; ++r) v[r] = pmul(v[r], twl[tb + r]);
    pdft8(v);
    if (si == nst - 1) break; /* v[r] = output t + r q */
    __syncthreads();
    const int so = pair_swz(((t >> lNs) << (lNs + 3)) + k);
#pragma unroll
    for (int r = 0; r < 8; ++r) bw[pair_at(so, r << lNs)] = pair_pack(v[r]);
    Ns <<= 3, lNs += 3;
  }
  float2 *const dp = ot.rpp ? reinterpret_cast<float2 *>(ot.p[row / ot.rpp]) + (row % ot.rpp) * fp.orow : out + row * fp.orow;
  const unsigned g = g0 + 2 * p, ostr = (unsigned)fp.ostr, qs = (unsigned)q * ostr;
  float2 *const op = dp + g * fp.oseq + t * ostr, *const oq = op + fp.oseq;
  const bool both = Ld::kOwnOut || !TOUT && fp.oseq == 1 && ((uintptr_t)dp & 15) == 0; /* (g and ostr are even) */
  Pair a{};
  if (fp.twiddle_post) {
    const float2 x = post(g * (unsigned)t), y = post((g + 1) * (unsigned)t);
    a = {make_float2(x.x, y.x), make_float2(x.y, y.y)};
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    Pair x = v[r];
    if (fp.twiddle_post) {
      const Pair w = pair_unpack(twq[p * 9 + r]), c = pmul(a, w.re, w.im, make_float2(-w.im.x, -w.im.y));
      x = pmul(x, c.re, c.im, make_float2(-c.im.x, -c.im.y));
    }
    if (fp.conj_out) x.im.x = -x.im.x, x.im.y = -x.im.y;
    if (both) {
      *reinterpret_cast<float4 *>(op + r * qs) = make_float4(x.re.x, x.im.x, x.re.y, x.im.y);
    } else {
      op[r * qs] = make_float2(x.re.x, x.im.x);
      oq[r * qs] = make_float2(x.re.y, x.im.y);
    }
  }
}
