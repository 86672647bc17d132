/*
 * FP32 row contractions of the FMM tree and leaf on the CUDA cores, sm_100a: out[r][c] = sum_k A(r, k)
 * B[k][c] over many rows r (section, re/im plane, box) with a small operator B.
 *
 * Bound: the shared-memory port next to the FMA units.  A 16-byte shared load costs an SM 2 to 3 cycles
 * a warp, an fma.rn.f32x2 half a cycle, so a thread's tile is 8 rows x 4 columns: 12 loads for 64
 * packed FMAs (4 or 2 rows where a level has too few to fill the device).  K goes in pairs (even-k and odd-k partial sums side by side), so that an A row's pairs
 * come as they lie in memory and the operator's as k_tree_ops lays them out (EngF32).  A block stages
 * the expansions and samples of a run of boxes once, halo boxes included: a neighbour's segment of K
 * is another row of the same shared array.  The operator of a level (or section) is staged before the
 * wait for the kernel that made the rows, and kept for all of a block's tiles.
 *
 * Measured against the general row kernels, the direct leaf and more levels in the one-warp-a-row
 * coarse tree (us, FP32, b = 32, P = 64): 2^24, 24 terms: M2L 1010 -> 309, M2M 249 -> 123, leaf 353 -> 250;
 * 2^20, 20 terms: M2L 64 -> 33, leaf 35 -> 25, coarse levels 57 -> 25, the transform 214 -> 128.  At 2^24
 * the M2L runs at 40% of the FMA rate, the leaf at 43%: 12 warps an SM hide the loads and barriers
 * between tiles only in part; the small levels of 2^20 are bound by their launches (3 to 4 us each).
 *
 * An output's sum runs over k in order whatever the tile, so a transform has the same bits with the
 * tiles that suit one transform and with those that suit a batch.
 */
#pragma once

/* A tile is R consecutive rows (a power of two): part of one plane, or whole planes.  Shared arrays
 * hold `pre` halo rows before and `post` after each plane's (or part's) rows. */
struct Tile32 {
  long r0;             /* first row */
  int valid, lnb, nbt; /* rows in it; log2 of, and the rows of a plane in the tile */
};

/* cp.async of V floats (1, 2), and the rest of rows32_copy for rows that are no multiple of 4 values: copies of
 * 8 bytes for even lengths, of 4 for odd ones.  All asynchronous: through registers a tile waited for each
 * load in turn and M2M and the leaf lost to the general kernels (2^22, P = 64, b = 16, us M2M, M2L, leaf: 9 terms 122,
 * 176, 93 -> 50, 90, 60, the general kernels 84, 207, 64; 10 terms 122, 177, 94 -> 45, 78, 56). */
template <int V> __device__ __forceinline__ void cp_async_f(uint32_t dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" : : "r"(dst), "l"(src), "n"(4 * V) : "memory");
}
template <int V>
__device__ __forceinline__ void rows32_copy_by(float *dst, int pitch, const float *__restrict__ src, int first, int count, int mask,
                                               int len) {
  const int step = blockDim.x >> 3, np = rows_kpad(len);
  for (int c = V * (threadIdx.x & 7); c < np; c += 8 * V)
    for (int j = threadIdx.x >> 3; j < count; j += step) {
      float *const d = dst + j * pitch + c;
      if (c < len) cp_async_f<V>(tc::smem_addr(d), src + (unsigned)(((first + j) & mask) * len) + c);
      else
#pragma unroll
        for (int v = 0; v < V; ++v) d[v] = 0.f;
    }
}
/* `count` rows of len values, from row `first` on (wrapping at mask + 1) of the strip src, into shared
 * rows of pitch; zeros up to a multiple of 4.  Eight lanes a row. */
__device__ __forceinline__ void rows32_copy(float *dst, int pitch, const float *__restrict__ src, int first, int count,
                                            int mask, int len) {
  const int c8 = threadIdx.x & 7, step = blockDim.x >> 3;
  if ((len & 3) == 0) {
    for (int c = 4 * c8; c < len; c += 32) {
      uint32_t d = tc::smem_addr(dst) + 4u * ((threadIdx.x >> 3) * pitch + c);
      const float *const g = src + c;
      for (int j = threadIdx.x >> 3; j < count; j += step, d += 4u * step * pitch)
        tc::cp_async16(d, g + (unsigned)(((first + j) & mask) * len));
    }
  } else if ((len & 1) == 0) {
    rows32_copy_by<2>(dst, pitch, src, first, count, mask, len);
  } else {
    rows32_copy_by<1>(dst, pitch, src, first, count, mask, len);
  }
}

/* Problems: arrays of the tile (stage), rows of a thread and outputs (dst).  aoff gives a row's places in
 * the first array (segment 0) and in the second (the others); segment s of parity par lies soff further,
 * the next row of the plane astep. */
struct R32M2L { /* child level l, one row per parent box: psi[B]; phi[2B-2], [2B+2], [2B+3] / [2B-2], [2B-1], [2B+3] */
  static constexpr int NSEG = 4, NPAR = 2;
  static constexpr bool kLeaf = false;
  const float *psi_par, *phi, *op;
  float *out;
  long rows;
  int T, lpar;
  __host__ __device__ int lplane() const { return lpar; }
  __host__ __device__ int ncol() const { return T; }
  __host__ __device__ int smem(int R) const {
    const int nbt = R < (1 << lpar) ? R : 1 << lpar;
    return (R + R / nbt * (2 * nbt + 4)) * tree_pitch(rows_kpad(T));
  }
  __device__ void stage(float *A, int R, const Tile32 &t, int) const {
    const int q = tree_pitch(rows_kpad(T));
    rows32_copy(A, q, psi_par + t.r0 * T, 0, t.valid, ~0, T);
    const long pl0 = t.r0 >> lpar;
    const int b0 = (int)(t.r0 & ((1L << lpar) - 1)), mask = (2 << lpar) - 1;
    for (int p = 0; p < t.valid >> t.lnb; ++p)
      rows32_copy(A + (R + p * (2 * t.nbt + 4)) * q, q, phi + ((pl0 + p) << (lpar + 1)) * T, 2 * b0 - 2, 2 * t.nbt + 4, mask, T);
  }
  __device__ void aoff(int R, const Tile32 &t, int r, int (&o)[2]) const {
    const int q = tree_pitch(rows_kpad(T)), p = r >> t.lnb, i = r & (t.nbt - 1);
    o[0] = r * q, o[1] = (R + p * (2 * t.nbt + 4) + 2 * i + 2) * q;
  }
  __device__ int astep(int s) const { return (s ? 2 : 1) * tree_pitch(rows_kpad(T)); }
  __device__ int soff(int s, int par) const {
    return (s == 0 ? 0 : s == 1 ? -2 : s == 2 ? (par ? -1 : 2) : 3) * tree_pitch(rows_kpad(T));
  }
  __device__ int len(int) const { return rows_kpad(T); }
  __device__ int bofs(int s, int par) const { return (par * 4 + s) * tree_blk<EngF32>(T); }
  __device__ float *dst(const Tile32 &t, int r, int par, int) const { return out + (2 * (t.r0 + r) + par) * T; }
};

struct R32M2M { /* parent level: the child pair */
  static constexpr int NSEG = 2, NPAR = 1;
  static constexpr bool kLeaf = false;
  const float *child, *op;
  float *out;
  long rows;
  int T;
  __host__ __device__ int lplane() const { return 62; }
  __host__ __device__ int ncol() const { return T; }
  __host__ __device__ int smem(int R) const { return 2 * R * tree_pitch(rows_kpad(T)); }
  __device__ void stage(float *A, int, const Tile32 &t, int) const {
    rows32_copy(A, tree_pitch(rows_kpad(T)), child + 2 * t.r0 * T, 0, 2 * t.valid, ~0, T);
  }
  __device__ void aoff(int, const Tile32 &, int r, int (&o)[2]) const { o[0] = o[1] = 2 * r * tree_pitch(rows_kpad(T)); }
  __device__ int astep(int) const { return 2 * tree_pitch(rows_kpad(T)); }
  __device__ int soff(int s, int) const { return s * tree_pitch(rows_kpad(T)); }
  __device__ int len(int) const { return rows_kpad(T); }
  __device__ int bofs(int s, int) const { return s * tree_blk<EngF32>(T); }
  __device__ float *dst(const Tile32 &t, int r, int, int) const { return out + (t.r0 + r) * T; }
};

struct R32S2M { /* leaf multipoles: a row's b samples (batch z = transform) */
  static constexpr int NSEG = 1, NPAR = 1;
  static constexpr bool kLeaf = false;
  const float *xt, *op;
  float *out;
  long rows, M;
  int T, b, P;
  __host__ __device__ int lplane() const { return 62; }
  __host__ __device__ int ncol() const { return T; }
  __host__ __device__ int smem(int R) const { return R * tree_pitch(b); }
  __device__ void stage(float *A, int, const Tile32 &t, int z) const {
    rows32_copy(A, tree_pitch(b), xt + (2L * P * z + 2) * M + t.r0 * b, 0, t.valid, ~0, b);
  }
  __device__ void aoff(int, const Tile32 &, int r, int (&o)[2]) const { o[0] = o[1] = r * tree_pitch(b); }
  __device__ int astep(int) const { return tree_pitch(b); }
  __device__ int soff(int, int) const { return 0; }
  __device__ int len(int) const { return b; }
  __device__ int bofs(int, int) const { return 0; }
  __device__ float *dst(const Tile32 &t, int r, int, int z) const { return out + ((long)z * rows + t.r0 + r) * T; }
};

/* Leaf of section z + 1 (RowsLeaf): psi[box], x[box - 1], x[box + 1] and, its weights reach P / pi, last
 * x[box]; and the half-shifted first points of sections from P/2 on. */
struct R32Leaf {
  static constexpr int NSEG = 4, NPAR = 1;
  static constexpr bool kLeaf = true;
  const float *psi_n, *xt, *op, *evalmh, *cot;
  float *u;
  long rows, M, s;
  int T, b, log2s, P;
  __device__ long plane(long r, int z) const { return (r >> (log2s + 1)) * 2 * (P - 1) + 2L * z + ((r >> log2s) & 1); }
  __host__ __device__ int lplane() const { return log2s; }
  __host__ __device__ int ncol() const { return b; }
  __host__ __device__ int nbt(int R) const { return R < s ? R : (int)s; }
  __host__ __device__ int smem(int R) const {
    return R / nbt(R) * ((nbt(R) + 1) * tree_pitch(rows_kpad(T)) + (nbt(R) + 3) * tree_pitch(b));
  }
  __device__ int xbase(int R, const Tile32 &t) const { return (R >> t.lnb) * (t.nbt + 1) * tree_pitch(rows_kpad(T)); }
  __device__ void stage(float *A, int R, const Tile32 &t, int z) const {
    const int q = tree_pitch(rows_kpad(T)), xq = tree_pitch(b);
    const int b0 = (int)(t.r0 & (s - 1)), mask = (int)s - 1;
    for (int p = 0; p < t.valid >> t.lnb; ++p) {
      const long r = t.r0 + ((long)p << t.lnb), pl = plane(r, z);
      rows32_copy(A + p * (t.nbt + 1) * q, q, psi_n + pl * s * T, b0 - 1, t.nbt + 1, mask, T);
      rows32_copy(A + xbase(R, t) + p * (t.nbt + 3) * xq, xq, xt + (pl + 2 * (r >> (log2s + 1)) + 2) * M, b0 - 2, t.nbt + 3, mask, b);
    }
  }
  __device__ void aoff(int R, const Tile32 &t, int r, int (&o)[2]) const {
    const int p = r >> t.lnb, i = r & (t.nbt - 1);
    o[0] = (p * (t.nbt + 1) + i + 1) * tree_pitch(rows_kpad(T));
    o[1] = xbase(R, t) + (p * (t.nbt + 3) + i + 2) * tree_pitch(b);
  }
  __device__ int astep(int sg) const { return tree_pitch(sg ? b : rows_kpad(T)); }
  __device__ int soff(int sg, int) const { return (sg == 1 ? -1 : sg == 2 ? 1 : 0) * tree_pitch(b); }
  __device__ int len(int sg) const { return sg == 0 ? rows_kpad(T) : b; }
  __device__ int bofs(int sg, int) const {
    return sg == 0 ? 0 : (rows_kpad(T) + (sg == 1 ? 0 : sg == 2 ? 2 * b : b)) * EngF32::npad(b);
  }
  __device__ float *dst(const Tile32 &t, int r, int, int z) const {
    return u + plane(t.r0 + r, z) * M + ((t.r0 + r) & (s - 1)) * b;
  }
};

constexpr int kRows32Threads = 128;
/* threads with rows of a tile: nrg (a power of two) by column groups of 4, at most a block's */
__host__ __device__ __forceinline__ int rows32_nrg(int ncx) {
  int n = 32;
  while (n * ncx > kRows32Threads) n >>= 1;
  return n;
}

/* Tiles of RT x nrg rows of batch blockIdx.y; the operator's nop values lie in shared memory, then (leaf)
 * the half-shift's weights and values, then the tile. */
template <class Prob, int RT>
__global__ void __launch_bounds__(kRows32Threads, 3) k_rows_f32(const __grid_constant__ Prob pb, int tiles, int nop, int nhw) {
  extern __shared__ __align__(16) unsigned char rows_raw[];
  float *const sop = reinterpret_cast<float *>(rows_raw);
  const int z = blockIdx.y, ncol = pb.ncol(), nc = (ncol + 3) >> 2, Np = 4 * nc, ncx = nc * Prob::NPAR;
  const int nrg = rows32_nrg(ncx), R = RT * nrg;
  float *const hw = sop + nop, *const hv = hw + nhw, *const A = hv + (Prob::kLeaf ? R : 0);
  tc::pdl_trigger();
  { /* plan constants: staged before the wait for the kernel that made the rows */
    const float *op = pb.op + (long)(Prob::kLeaf ? z : 0) * nop;
    for (int e = 4 * threadIdx.x; e < nop; e += 4 * blockDim.x) tc::cp_async16(tc::smem_addr(sop + e), op + e);
  }
  bool shifted = false;
  if constexpr (Prob::kLeaf) {
    shifted = 2 * (z + 1) >= pb.P;
    const int Tp = rows_kpad(pb.T);
    if (shifted)
      for (int e = threadIdx.x; e < nhw; e += blockDim.x)
        hw[e] = e < pb.T ? pb.evalmh[(long)z * pb.T + e] : e < Tp ? 0.f : pb.cot[(long)z * 4 * pb.b + e - Tp];
  }
  tc::pdl_wait();
  constexpr bool kOnePlane = RT > 2; /* a tile lies in one plane: its rows are evenly spaced */
  Tile32 t;
  t.lnb = min(pb.lplane(), __ffs(R) - 1), t.nbt = 1 << t.lnb;
  /* parities apart: 8 neighbouring lanes read one operator's columns and two or three rows, no bank twice */
  const int par = (int)threadIdx.x / (nrg * nc), rem = (int)threadIdx.x - par * nrg * nc, rg = rem / nc, cg = rem - rg * nc;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    t.r0 = (long)tile * R;
    t.valid = pb.rows - t.r0 < R ? (int)(pb.rows - t.r0) : R;
    if (tile != (int)blockIdx.x) __syncthreads(); /* the tile before is done with */
    pb.stage(A, R, t, z);
    tc::cp_async_wait_all();
    __syncthreads();
    if constexpr (Prob::kLeaf)
      if (shifted) { /* first points, from the box before: a thread a box */
        const int Tp = rows_kpad(pb.T), b = pb.b, q = tree_pitch(Tp), xq = tree_pitch(b);
        for (int r = threadIdx.x; r < R; r += blockDim.x) {
          int o[2];
          pb.aoff(R, t, r, o);
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          auto dot = [&](const float *a, const float *w, int n) {
#pragma unroll 2
            for (int k = 0; k < n; k += 4) {
              const float4 x = *reinterpret_cast<const float4 *>(a + k), y = *reinterpret_cast<const float4 *>(w + k);
              v.x = fmaf(x.x, y.x, v.x), v.y = fmaf(x.y, y.y, v.y), v.z = fmaf(x.z, y.z, v.z), v.w = fmaf(x.w, y.w, v.w);
            }
          };
          dot(A + o[0] - q, hw, Tp);
          for (int g = 0; g < 3; ++g) dot(A + o[1] + (g - 2) * xq, hw + Tp + g * b, b);
          hv[r] = (v.x + v.y) + (v.z + v.w);
        }
        __syncthreads();
      }
    if (par >= Prob::NPAR) continue;
    float2 acc[RT][4];
    int o[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int s = 0; s < Prob::NSEG; ++s) {
      const int K = pb.len(s), so = pb.soff(s, par);
      const int step = nrg * pb.astep(s);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        if (kOnePlane && i > 0) {
          o[i] = o[i - 1] + step;
        } else {
          int o2[2];
          pb.aoff(R, t, rg + i * nrg, o2);
          o[i] = (s == 0 ? o2[0] : o2[1]) + so;
        }
      }
      const float *bp = sop + pb.bofs(s, par) + 4 * cg;
#pragma unroll 1
      for (int k = 0; k < K; k += 4, bp += 4 * Np) {
        const float4 b0 = *reinterpret_cast<const float4 *>(bp), b1 = *reinterpret_cast<const float4 *>(bp + Np);
        const float4 b2 = *reinterpret_cast<const float4 *>(bp + 2 * Np), b3 = *reinterpret_cast<const float4 *>(bp + 3 * Np);
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          const float4 a = *reinterpret_cast<const float4 *>(A + o[i] + k);
          const float2 a0 = make_float2(a.x, a.y), a1 = make_float2(a.z, a.w);
          acc[i][0] = ffma2(a0, make_float2(b0.x, b0.y), acc[i][0]);
          acc[i][1] = ffma2(a0, make_float2(b0.z, b0.w), acc[i][1]);
          acc[i][2] = ffma2(a0, make_float2(b1.x, b1.y), acc[i][2]);
          acc[i][3] = ffma2(a0, make_float2(b1.z, b1.w), acc[i][3]);
          acc[i][0] = ffma2(a1, make_float2(b2.x, b2.y), acc[i][0]);
          acc[i][1] = ffma2(a1, make_float2(b2.z, b2.w), acc[i][1]);
          acc[i][2] = ffma2(a1, make_float2(b3.x, b3.y), acc[i][2]);
          acc[i][3] = ffma2(a1, make_float2(b3.z, b3.w), acc[i][3]);
        }
      }
    }
    const bool pairs = (ncol & 1) == 0, c2 = Np / 2 + 2 * cg < ncol;
    float *d = pb.dst(t, rg, par, z) + 2 * cg;
    const int step = nrg * Prob::NPAR * ncol;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = rg + i * nrg;
      if (!kOnePlane && i > 0) d = pb.dst(t, r, par, z) + 2 * cg;
      float v0 = acc[i][0].x + acc[i][0].y;
      const float v1 = acc[i][1].x + acc[i][1].y, v2 = acc[i][2].x + acc[i][2].y, v3 = acc[i][3].x + acc[i][3].y;
      if constexpr (Prob::kLeaf)
        if (shifted && cg == 0) v0 = 2 * (z + 1) == pb.P ? 0.5f * (v0 + hv[r]) : hv[r];
      if (r < t.valid) {
        if (pairs) { /* the row starts on a pair: rows are ncol values apart */
          if (2 * cg < ncol) *reinterpret_cast<float2 *>(d) = make_float2(v0, v1);
          if (c2) *reinterpret_cast<float2 *>(d + Np / 2) = make_float2(v2, v3);
        } else {
          if (2 * cg < ncol) d[0] = v0;
          if (2 * cg + 1 < ncol) d[1] = v1;
          if (c2) d[Np / 2] = v2;
          if (Np / 2 + 2 * cg + 1 < ncol) d[Np / 2 + 1] = v3;
        }
      }
      if (kOnePlane) d += step;
    }
  }
}
