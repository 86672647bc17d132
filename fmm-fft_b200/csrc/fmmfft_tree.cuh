/*
 * The FMM of a small section in one block, sm_100a: x -> u (reference src/fmmfft.c:419-954) with every
 * tree level in shared memory.
 *
 * Every section of the transform is a tree of its own from its samples to its field, so sections of
 * up to a few thousand points need no launch between levels, no planar copy of the samples and no
 * pass for their sums; which plans take it is tree_setup's rule.  Here a stage costs two
 * block barriers, and its contraction is blk_gemm: out[row][c] = sum_k A(row, k) B[k][c], A rows and B
 * in shared memory, a thread (FP32) a register tile of the output, a warp (FP64) tiles of the FP64
 * matrix instruction.  Bound by latency: a stage of a small section is a chain of a few hundred
 * instructions a warp (1500 to 6000 cycles), whether a block runs alone or beside four others (16
 * transforms of 2^16, P = 64, 20 terms: 37 k instructions a warp-block, 35% of the issue slots).
 *
 * An output's sum runs over k in order whatever the tile, so a transform has the same bits with
 * the tile sizes that suit one transform and with those that suit a batch.
 */
#pragma once

/* Pitch of a shared row of n values, 4 mod 8: the rows a warp reads at one k (8 rows x 4 values for
 * the matrix instruction, 16-byte vectors of neighbouring rows otherwise) lie in different banks. */
__host__ __device__ __forceinline__ int tree_pitch(int n) { return ((n + 3) & ~7) + 4; }

/* The arithmetic of a plan's tree kernel.  An operator block of K rows (a multiple of 4) and np columns
 * holds element (k, c) at idx, as the instructions read it; kc is its inverse. */
struct EngF32 { /* K interleaved by two, for fma.rn.f32x2: the pair holds the even-k and the odd-k partial sum */
  using R = float;
  static constexpr int V = 4; /* values of a 16-byte load */
  __host__ __device__ static int npad(int N) { return (N + 3) & ~3; }
  __device__ static void kc(long e, int np, int &k, int &c) {
    const int q = (int)(e >> 1);
    k = q / np * 2 + (int)(e & 1), c = q % np;
  }
};
struct EngF64 { /* B fragments of mma.m8n8k4 (fmmfft_rows.cuh) */
  using R = double;
  static constexpr int V = 2;
  __host__ __device__ static int npad(int N) { return rows_npad(N); }
  __device__ static void kc(long e, int np, int &k, int &c) { rows_kc(e, np, k, c); }
};
template <typename R> struct TreeEng;
template <> struct TreeEng<float> { using E = EngF32; };
template <> struct TreeEng<double> { using E = EngF64; };

template <class E> __host__ __device__ __forceinline__ int tree_blk(int T) { return rows_kpad(T) * E::npad(T); }
template <class E> __host__ __device__ __forceinline__ int tree_nleaf(int T, int b) { return (rows_kpad(T) + 3 * b) * E::npad(b); }

/* Operators in the plan's memory, back to back: S2M (b x T), then T x T blocks: M2M of the parent
 * levels 2 .. n-1 (left, right child), M2L of the child levels 3 .. n (left child: psi, phi c-2, c+2,
 * c+3; right child: psi, phi c-3, c-2, c+2), top flip; then the sections' leaf operators: psi (T x b)
 * and the boxes before, at and after (b x b). */
template <class E> struct TreeOps {
  const typename E::R *s2m, *m2m, *m2l, *top, *leaf;
  __host__ __device__ void set(const typename E::R *p, int T, int b, int nl) {
    const long blk = tree_blk<E>(T);
    s2m = p, m2m = s2m + (long)b * E::npad(T), m2l = m2m + nl * 2 * blk, top = m2l + nl * 8 * blk, leaf = top + blk;
  }
};
template <class E> static long tree_nops(long P, long T, long b, long nl) {
  return b * E::npad((int)T) + (nl * 10 + 1) * tree_blk<E>((int)T) + (P - 1) * tree_nleaf<E>((int)T, (int)b);
}
/* The operators laid out on the device from the plan's own tables; zero beyond a table. */
template <class E>
__global__ void k_tree_ops(typename E::R *__restrict__ out, const typename E::R *__restrict__ initch,
                           const typename E::R *__restrict__ bm2m, const typename E::R *__restrict__ bm2l,
                           const typename E::R *__restrict__ btop, const typename E::R *__restrict__ evalmT,
                           const typename E::R *__restrict__ cot, long total, int T, int b, int nl) {
  using R = typename E::R;
  const int Tp = rows_kpad(T), Tn = E::npad(T), bn = E::npad(b), blk = Tp * Tn;
  const long n_s2m = (long)b * Tn, n_m2m = n_s2m + (long)nl * 2 * blk, n_m2l = n_m2m + (long)nl * 8 * blk, n_top = n_m2l + blk,
             nlf = tree_nleaf<E>(T, b);
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    int k, c;
    R v = 0;
    if (e < n_s2m) {
      E::kc(e, Tn, k, c);
      if (k < b && c < T) v = initch[k * T + c];
    } else if (e < n_top) {
      const long q = e < n_m2m ? e - n_s2m : e < n_m2l ? e - n_m2m : e - n_m2l, g = q / blk;
      E::kc(q - g * blk, Tn, k, c);
      if (k < T && c < T) {
        if (e < n_m2m) {
          v = bm2m[((g >> 1) * 2 * T + (g & 1) * T + k) * T + c];
        } else if (e < n_m2l) { /* rows psi, phi[2B-2], phi[2B-1], phi[2B+2], phi[2B+3] of the stacked operator */
          const int j = (int)(g & 7), right = j >> 2, seg = (j & 3) + ((j & 3) >= (right ? 3 : 2));
          v = bm2l[((g >> 3) * 5 * T + seg * T + k) * 2 * T + right * T + c];
        } else {
          v = btop[k * T + c];
        }
      }
    } else {
      const long q = e - n_top, z = q / nlf, r = q - z * nlf;
      if (r < (long)Tp * bn) {
        E::kc(r, bn, k, c);
        if (k < T && c < b) v = evalmT[(z * T + k) * b + c];
      } else {
        const long r2 = r - (long)Tp * bn, seg = r2 / ((long)b * bn);
        E::kc(r2 - seg * b * bn, bn, k, c);
        if (c < b) v = cot[z * 4 * b + seg * b + k + b - c];
      }
    }
    out[e] = v;
  }
}

/* ------------------------------------------------------------------------ contraction */
/* One stage: out(row, par)[c] = sum over segments g of sum_k A_g(row, par)[k] B_par,g[k][c].  Rows are
 * (plane, box), 2^rsh boxes a plane; segment g of row (pl, i) is row (pl, (mul i + par (mul - 1) +
 * d[par]) mod 2^csh) of a shared array of expansions or samples.  Every stage has this form, so that
 * one copy of the loops serves all of them: a small transform runs each stage once, and its
 * instructions would come from memory each time. */
struct TreeSeg {
  int base, pitch, csh, mul, d[2], len, bofs[2]; /* A array, K (a multiple of 4), operator blocks */
};
struct TreeStage {
  TreeSeg seg[4];
  int nseg, rows, rsh, ncol, npar;
  unsigned rcp; /* ceil(2^32 / (column groups times npar)), 0 for 1: a tile's row group without a division */
  int so;       /* shared rows of the result (pitch Tq), or -1 */
  int gn;       /* values of a result row in global memory */
  int lv;       /* the level it belongs to, 0: the field */
  int op, nop;  /* its operator: place in shared memory, values */
};

__device__ __forceinline__ int tree_aoff(const TreeSeg &g, int hi, int lo, int par) {
  const int c = lo * g.mul + par * (g.mul - 1) + g.d[par];
  return g.base + ((hi << g.csh) + (c & ((1 << g.csh) - 1))) * g.pitch;
}

/* FP32: a thread takes TR rows and the columns 2 cg, 2 cg + 1, Np/2 + 2 cg, + 1.  An A row's pairs
 * come as they lie in memory, so no operand is duplicated or moved.  The shared-memory port bounds
 * it: 8 16-byte loads for the 64 FMAs of a 4-row tile, 5 for the 16 of a one-row tile, so tiles are
 * large where blocks fill the device, whatever threads that leaves idle, and small where a few blocks
 * run alone. */
template <int TR, class Out>
__device__ __forceinline__ void fma_gemm(const float *__restrict__ sm, const TreeStage &st, Out out) {
  const int rows = st.rows, nc = (st.ncol + 3) >> 2, Np = 4 * nc, ncx = nc * st.npar, nrg = (rows + TR - 1) / TR;
  const int rsh = st.rsh, rmask = (1 << rsh) - 1, nseg = st.nseg;
  const unsigned rcp = st.rcp;
  for (int it = threadIdx.x; it < nrg * ncx; it += blockDim.x) {
    const int rg = rcp ? (int)__umulhi((unsigned)it, rcp) : it, cx = it - rg * ncx, par = cx >= nc, cg = cx - par * nc;
    float2 acc[TR][4];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int g = 0; g < nseg; ++g) {
      const TreeSeg &sg = st.seg[g];
      int ao[TR];
#pragma unroll
      for (int i = 0; i < TR; ++i) {
        const int r = rg + i * nrg < rows ? rg + i * nrg : rows - 1;
        ao[i] = tree_aoff(sg, r >> rsh, r & rmask, par);
      }
      const int K = sg.len;
      const float *bp = sm + sg.bofs[par] + 4 * cg;
#pragma unroll (TR == 1 ? 4 : 2)
      for (int k = 0; k < K; k += 4, bp += 4 * Np) {
        float4 a[TR];
#pragma unroll
        for (int i = 0; i < TR; ++i) a[i] = *reinterpret_cast<const float4 *>(sm + ao[i] + k);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float4 b0 = *reinterpret_cast<const float4 *>(bp + p * 2 * Np);
          const float4 b1 = *reinterpret_cast<const float4 *>(bp + (2 * p + 1) * Np);
#pragma unroll
          for (int i = 0; i < TR; ++i) {
            const float2 av = p ? make_float2(a[i].z, a[i].w) : make_float2(a[i].x, a[i].y);
            acc[i][0] = ffma2(av, make_float2(b0.x, b0.y), acc[i][0]);
            acc[i][1] = ffma2(av, make_float2(b0.z, b0.w), acc[i][1]);
            acc[i][2] = ffma2(av, make_float2(b1.x, b1.y), acc[i][2]);
            acc[i][3] = ffma2(av, make_float2(b1.z, b1.w), acc[i][3]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      const int r = rg + i * nrg;
      if (r < rows) {
        out(r, par, 2 * cg, acc[i][0].x + acc[i][0].y, acc[i][1].x + acc[i][1].y);
        if (Np / 2 + 2 * cg < st.ncol) out(r, par, Np / 2 + 2 * cg, acc[i][2].x + acc[i][2].y, acc[i][3].x + acc[i][3].y);
      }
    }
  }
}

/* FP64: a warp takes RT tiles of 8 rows and one of 8 columns; lane (g, t) = (lane / 4, lane % 4) holds
 * A (row g, k = t), B (k = t, column g) and C (row g, columns 2t, 2t + 1). */
template <int RT, class Out>
__device__ __forceinline__ void dmma_gemm(const double *__restrict__ sm, const TreeStage &st, Out out) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rows = st.rows, nt = (st.ncol + 7) >> 3, ncx = nt * st.npar, nrg = (rows + 8 * RT - 1) / (8 * RT);
  const int rsh = st.rsh, rmask = (1 << rsh) - 1, nseg = st.nseg;
  const unsigned rcp = st.rcp;
  for (int it = threadIdx.x >> 5; it < nrg * ncx; it += blockDim.x >> 5) {
    const int rg = rcp ? (int)__umulhi((unsigned)it, rcp) : it, cx = it - rg * ncx, par = cx >= nt, j0 = cx - par * nt;
    double acc[RT][2];
    int ao[4][RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r0 = (rg * RT + i) * 8 + g, r = r0 < rows ? r0 : rows - 1, hi = r >> rsh, lo = r & rmask;
#pragma unroll
      for (int s = 0; s < 4; ++s) ao[s][i] = tree_aoff(st.seg[s], hi, lo, par) + t;
      acc[i][0] = acc[i][1] = 0.0;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (s >= nseg) break;
      const double *bp = sm + st.seg[s].bofs[par] + j0 * 32 + lane;
      const int k4n = st.seg[s].len >> 2;
#pragma unroll 4
      for (int k4 = 0; k4 < k4n; ++k4) {
        const double bv = bp[k4 * nt * 32];
#pragma unroll
        for (int i = 0; i < RT; ++i) mma_f64(acc[i], sm[ao[s][i] + 4 * k4], bv);
      }
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = (rg * RT + i) * 8 + g, c = j0 * 8 + 2 * t;
      if (r < rows && c < st.ncol) out(r, par, c, acc[i][0], acc[i][1]);
    }
  }
}

/* The stage in the largest tile that gives `want` threads work; out(row, par, c, v0, v1) takes the
 * columns c and c + 1 (c even). */
template <class Out> __device__ __forceinline__ void blk_gemm(const float *__restrict__ sm, const TreeStage &st, int want, Out out) {
  const int t1 = st.rows * ((st.ncol + 3) >> 2) * st.npar; /* one-row tiles */
  if (t1 >= 4 * want) fma_gemm<4>(sm, st, out);
  else if (t1 >= 2 * want) fma_gemm<2>(sm, st, out);
  else fma_gemm<1>(sm, st, out);
}
template <class Out> __device__ __forceinline__ void blk_gemm(const double *__restrict__ sm, const TreeStage &st, int want, Out out) {
  if (((st.rows + 31) >> 5) * ((st.ncol + 7) >> 3) * st.npar * 32 >= want) dmma_gemm<4>(sm, st, out);
  else dmma_gemm<1>(sm, st, out);
}

/* Issue the copy of n values (n a multiple of V, both sides 16-byte aligned) into shared memory. */
template <typename R> __device__ __forceinline__ void tree_stage(R *dst, const R *__restrict__ src, int n) {
  constexpr int V = 16 / (int)sizeof(R);
  const uint32_t d = tc::smem_addr(dst);
  for (int e = threadIdx.x * V; e < n; e += blockDim.x * V) tc::cp_async16(d + (uint32_t)(e * sizeof(R)), src + e);
}
__device__ __forceinline__ void tree_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void tree_wait() {
  asm volatile("cp.async.wait_group %0;" : : "n"(N) : "memory");
}

/* Two neighbouring columns of a row of n values in global memory, and in a shared row (c even). */
template <typename R> __device__ __forceinline__ void tree_put2(R *__restrict__ row, int n, int c, R v0, R v1) {
  if ((n & 1) == 0) {
    if (c < n) {
      typename cplx<R>::T v;
      v.x = v0, v.y = v1;
      *reinterpret_cast<typename cplx<R>::T *>(row + c) = v;
    }
  } else {
    if (c < n) row[c] = v0;
    if (c + 1 < n) row[c + 1] = v1;
  }
}
template <typename R> __device__ __forceinline__ void tree_sput2(R *__restrict__ p, R v0, R v1) {
  typename cplx<R>::T v;
  v.x = v0, v.y = v1;
  *reinterpret_cast<typename cplx<R>::T *>(p) = v;
}

/* ------------------------------------------------------------------------ a whole small section */
template <class E> struct TreeArgs {
  using R = typename E::R;
  const typename cplx<R>::T *x;
  R *xt;
  typename cplx<R>::T *ssum;
  R *phi, *psi, *u;
  TreeOps<E> op;
  const R *evalmh, *cot;
  const TreeStage *stages; /* tree_stages of this form */
  long M, S1e;
  int P, T, b, n, conj;
  int resident; /* every operator has a place of its own, copied at the start; else one buffer for all in turn */
  int want;     /* threads that a stage's tiles should keep busy (smaller tiles for few blocks) */
  InTab xin;
};

/* Values of the largest operator (M2L's where there is one), and of the operators' place in shared memory */
template <class E> __host__ __device__ __forceinline__ int tree_opn(int T, int b, int n) {
  int m = (n > 2 ? 8 : 1) * tree_blk<E>(T);
  if (tree_nleaf<E>(T, b) > m) m = tree_nleaf<E>(T, b);
  if (b * E::npad(T) > m) m = b * E::npad(T);
  return m;
}
template <class E> __host__ __device__ __forceinline__ int tree_op_area(int T, int b, int n, int resident) {
  return resident ? b * E::npad(T) + (10 * (n - 2) + 1) * tree_blk<E>(T) + tree_nleaf<E>(T, b) : tree_opn<E>(T, b, n);
}
constexpr int kTreeMaxLevel = 12;                             /* n <= 12 */
constexpr int kTreeStages = 2 * (kTreeMaxLevel - 2) + 3; /* S2M, M2M n-1 .. 2, top flip, M2L 3 .. n, leaf */
constexpr int kTreeRed = 16;                                  /* values of the section sum's reduction */

/* Shared layout of a block, in values: operators (all of them, or a buffer for one), phi
 * levels 2 .. n of both planes, two levels of psi, samples, the half-shift column and its values, the
 * section sum's reduction; the stage table follows. */
template <class E> struct TreeLay {
  int ph, ps0, ps1, x, h, hv, red, end;
  __host__ __device__ TreeLay(int T, int b, int n, int resident) {
    const int Tq = tree_pitch(rows_kpad(T)), s = 1 << n;
    ph = tree_op_area<E>(T, b, n, resident);
    ps0 = ph + 2 * (2 * s - 4) * Tq, ps1 = ps0 + 2 * s * Tq, x = ps1 + s * Tq, h = x + 2 * s * tree_pitch(b);
    hv = h + rows_kpad(T) + 3 * b, red = hv + 2 * s, end = red + kTreeRed;
  }
};
template <class E> static size_t tree_smem(int T, int b, int n, int resident) {
  return sizeof(typename E::R) * (size_t)TreeLay<E>(T, b, n, resident).end + sizeof(TreeStage) * (2 * (n - 2) + 3);
}

/* The stages of a plan's k_tree, in the shared offsets of one of its two forms. */
template <class E> static void tree_stages(TreeStage *out, int T, int b, int n, int resident) {
  const int Tp = rows_kpad(T), Tq = tree_pitch(Tp), Tn = E::npad(T), blk = Tp * Tn, bn = E::npad(b), xq = tree_pitch(b);
  const int s = 1 << n, ns = 2 * (n - 2) + 3, a_top = b * Tn + 10 * (n - 2) * blk;
  const TreeLay<E> lay(T, b, n, resident);
  auto phl = [&](int l) { return lay.ph + 2 * ((1 << l) - 4) * Tq; };
  auto psl = [&](int l) { return ((n - l) & 1) ? lay.ps1 : lay.ps0; };
  for (int i = 0; i < ns; ++i) {
    TreeStage g{};
    const int at = i == 0 ? 0 : i <= n - 2 ? b * Tn + 2 * (n - i - 2) * blk : i == n - 1 ? a_top
                   : i < ns - 1 ? b * Tn + 2 * (n - 2) * blk + 8 * (i - n) * blk : a_top + blk;
    g.op = resident ? at : 0;
    auto seg = [&](int base, int pitch, int csh, int mul, int d0, int d1, int len, int b0, int b1) {
      g.seg[g.nseg++] = TreeSeg{base, pitch, csh, mul, {d0, d1}, len, {g.op + b0, g.op + b1}};
    };
    g.npar = 1, g.ncol = Tp, g.gn = T, g.lv = 2;
    if (i == 0) { /* S2M */
      g.lv = n, g.rows = 2 * s, g.rsh = n, g.so = phl(n), g.nop = b * Tn;
      seg(lay.x, xq, n, 1, 0, 0, b, 0, 0);
    } else if (i <= n - 2) { /* M2M of the child pair */
      const int l = n - i;
      g.lv = l, g.rows = 2 << l, g.rsh = l, g.so = phl(l), g.nop = 2 * blk;
      seg(phl(l + 1), Tq, l + 1, 2, 0, 0, Tp, 0, 0), seg(phl(l + 1), Tq, l + 1, 2, 1, 1, Tp, blk, blk);
    } else if (i == n - 1) { /* top flip: psi_2[c] from phi_2[c + 2 mod 4] */
      g.rows = 8, g.rsh = 2, g.so = psl(2), g.nop = blk;
      seg(phl(2), Tq, 2, 1, 2, 2, Tp, 0, 0);
    } else if (i < ns - 1) { /* M2L + L2L: psi of the parent, phi of c - 2, c + 2, c + 3 / c - 3, c - 2, c + 2 */
      const int l = i - n + 3;
      g.lv = l, g.rows = 1 << l, g.rsh = l - 1, g.npar = 2, g.so = psl(l), g.nop = 8 * blk;
      seg(psl(l - 1), Tq, l - 1, 1, 0, 0, Tp, 0, 4 * blk);
      seg(phl(l), Tq, l, 2, -2, -3, Tp, blk, 5 * blk);
      seg(phl(l), Tq, l, 2, 2, -2, Tp, 2 * blk, 6 * blk);
      seg(phl(l), Tq, l, 2, 3, 2, Tp, 3 * blk, 7 * blk);
    } else { /* leaf: psi, the boxes before, after and (its weights reach P / pi: last) at the row's */
      g.rows = 2 * s, g.rsh = n, g.ncol = b, g.so = -1, g.gn = b, g.lv = 0, g.nop = tree_nleaf<E>(T, b);
      seg(psl(n), Tq, n, 1, 0, 0, Tp, 0, 0);
      seg(lay.x, xq, n, 1, -1, -1, b, Tp * bn, 0);
      seg(lay.x, xq, n, 1, 1, 1, b, (Tp + 2 * b) * bn, 0);
      seg(lay.x, xq, n, 1, 0, 0, b, (Tp + b) * bn, 0);
    }
    const unsigned ncx = (unsigned)((sizeof(typename E::R) == 8 ? (g.ncol + 7) / 8 : (g.ncol + 3) / 4) * g.npar);
    g.rcp = ncx == 1 ? 0u : (unsigned)((0x100000000ull + ncx - 1) / ncx);
    out[i] = g;
  }
}

/* Section blockIdx.x of transform blockIdx.y; section 0, which has no field, only leaves its planar
 * copy and its sum.  The expansions also go to global memory (the stage views read them there). */
template <class E, int NT>
__global__ void __launch_bounds__(NT, NT == 128 ? 5 : 1) k_tree(const __grid_constant__ TreeArgs<E> a) {
  using R = typename E::R;
  using C = typename cplx<R>::T;
  constexpr int V = E::V;
  extern __shared__ __align__(16) unsigned char tree_raw[];
  R *const sm = reinterpret_cast<R *>(tree_raw);
  const int T = a.T, Tp = rows_kpad(T), Tq = tree_pitch(Tp), b = a.b, n = a.n, s = 1 << n, want = a.want;
  const int xq = tree_pitch(b), lb = __ffs(b) - 1, ns = 2 * (n - 2) + 3;
  const TreeLay<E> lay(T, b, n, a.resident);
  TreeStage *const stages = reinterpret_cast<TreeStage *>(sm + lay.end);
  const int sc = (int)blockIdx.x;
  const long tr = blockIdx.y, S1 = a.P - 1, M = a.M, pl0 = tr * 2 * S1 + 2L * (sc - 1);
  const bool shifted = 2 * sc >= a.P;
  const R *const leaf_op = a.op.leaf + (long)(sc - 1) * tree_nleaf<E>(T, b);
  /* the operator of stage i: the tree's lie back to back in the plan in level order, as in shared memory */
  auto stage_op = [&](int i) {
    const int blk = tree_blk<E>(T);
    const R *src = i == 0 ? a.op.s2m : i <= n - 2 ? a.op.m2m + (long)(n - i - 2) * 2 * blk
                   : i == n - 1 ? a.op.top : i < ns - 1 ? a.op.m2l + (long)(i - n) * 8 * blk : leaf_op;
    tree_stage<R>(sm + stages[i].op, src, stages[i].nop);
  };
  if (sc > 0) {
    { /* the stage table: whole 4-byte words, 8-byte aligned */
      const int nw = ns * (int)(sizeof(TreeStage) / 4);
      for (int e = threadIdx.x; e < nw; e += NT) reinterpret_cast<int *>(stages)[e] = reinterpret_cast<const int *>(a.stages)[e];
    }
    if (a.resident) { /* every operator, copied at once */
      tree_stage<R>(sm, a.op.s2m, b * E::npad(T) + (10 * (n - 2) + 1) * tree_blk<E>(T));
      tree_stage<R>(sm + b * E::npad(T) + (10 * (n - 2) + 1) * tree_blk<E>(T), leaf_op, tree_nleaf<E>(T, b));
    } else {
      tree_stage<R>(sm, a.op.s2m, b * E::npad(T));
    }
    tree_commit();
    if (shifted)
      for (int e = threadIdx.x; e < Tp + 3 * b; e += NT)
        sm[lay.h + e] = e < T ? a.evalmh[(long)(sc - 1) * T + e] : e < Tp ? R(0) : a.cot[(long)(sc - 1) * 4 * b + e - Tp];
  }
  { /* the section's samples and their sum (its order fixed by the section's size) */
    const C *x = (a.xin.n ? reinterpret_cast<const C *>(a.xin.p[tr]) : a.x + tr * M * a.P) + sc;
    for (int m0 = threadIdx.x; m0 < M; m0 += 8 * NT) {
      C v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (m0 + q * NT < M) v[q] = x[(long)(m0 + q * NT) * a.P];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int m = m0 + q * NT;
        if (m < M) {
          if (a.conj) v[q].y = -v[q].y;
          R *d = sm + lay.x + (m >> lb) * xq + (m & (b - 1));
          d[0] = v[q].x, d[s * xq] = v[q].y;
          if (sc == 0) a.xt[tr * 2 * a.P * M + m] = v[q].x, a.xt[(tr * 2 * a.P + 1) * M + m] = v[q].y;
        }
      }
    }
  }
  /* section sum, added up by the last warps while the first ones begin S2M: plane w / 8, eighth w % 8 */
  auto partial_sums = [&]() {
    for (int w = threadIdx.x >> 5; w < 16; w += NT / 32) {
      const int lane = threadIdx.x & 31;
      R t = 0;
      for (int m = (w & 7) * (int)(M >> 3) + lane; m < ((w & 7) + 1) * (int)(M >> 3); m += 32)
        t += sm[lay.x + (w >> 3) * s * xq + (m >> lb) * xq + (m & (b - 1))];
#pragma unroll
      for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) sm[lay.red + w] = t;
    }
  };
  auto final_sum = [&]() {
    if (threadIdx.x < 2) {
      R t = 0;
      for (int w = 0; w < 8; ++w) t += sm[lay.red + 8 * threadIdx.x + w];
      reinterpret_cast<R *>(a.ssum + tr * a.P + sc)[threadIdx.x] = t;
    }
  };
  if (sc == 0) {
    __syncthreads();
    partial_sums();
    __syncthreads();
    final_sum();
    return;
  }
  for (int i = 0; i < ns; ++i) {
    if (a.resident) {
      if (i == 0) tree_wait<0>();
      __syncthreads(); /* the stage before is written; i = 0: samples, operators and table are in place */
    } else {
      if (i > 0) {
        __syncthreads(); /* the stage before is written and done with the operator buffer */
        stage_op(i);
        tree_commit();
      }
      tree_wait<0>();
      __syncthreads(); /* this stage's operator is in place */
    }
    if (i == 0) partial_sums();
    if (i == 1) final_sum();
    const TreeStage &sg = stages[i];
    const bool leaf = i == ns - 1;
    if (leaf && shifted) { /* the half-shifted first point of each box, from the box before it: 8 lanes a box */
      const int ps = sg.seg[0].base;
      for (int base = threadIdx.x & ~31; base < 16 * s; base += NT) {
        const int it = base + (threadIdx.x & 31), r = it >> 3, pl = r >> n, j = r & (s - 1);
        R t = 0;
        if (it < 16 * s)
          for (int k = (it & 7) * V; k < Tp + 3 * b; k += 8 * V) {
            const int q = k - Tp, seg = q < b ? 0 : q < 2 * b ? 1 : 2;
            const int ao = k < Tp ? ps + (pl * s + ((j - 1) & (s - 1))) * Tq + k
                                  : lay.x + (pl * s + ((j - 2 + seg) & (s - 1))) * xq + q - seg * b;
#pragma unroll
            for (int v = 0; v < V; ++v) t = fma(sm[ao + v], sm[lay.h + k + v], t);
          }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (it < 16 * s && (it & 7) == 0) sm[lay.hv + r] = t;
      }
      __syncthreads();
    }
    R *const gbase = leaf ? a.u + pl0 * M
                          : (i <= n - 2 ? a.phi : a.psi) + lvl_off(sg.lv, a.S1e, T) + pl0 * (1L << sg.lv) * T;
    const int so = sg.so, gn = sg.gn, npar = sg.npar;
    blk_gemm(sm, sg, want, [&](int r, int par, int c, R v0, R v1) {
      const int row = r * npar + par;
      if (so >= 0) tree_sput2<R>(sm + so + row * Tq + c, v0, v1);
      else if (c == 0 && shifted) v0 = 2 * sc == a.P ? R(0.5) * (v0 + sm[lay.hv + row]) : sm[lay.hv + row];
      tree_put2<R>(gbase + (long)row * gn, gn, c, v0, v1);
    });
  }
}

/* ------------------------------------------------------------------------ the coarse levels of a large tree */
/* The levels of few boxes in one launch, a block an expansion plane (section, re/im, transform; planes are
 * independent at every level): M2M for parent levels Lm .. 2, the top flip, M2L + L2L for child levels
 * 3 .. Ll, each a stage of blk_gemm between two barriers.  phi of the level below comes from global
 * memory, every level made here goes there too (the row contractions and the debug views read it).  A
 * launch a level costs 3 to 4 us.  Bound by latency, like k_tree: us a launch, with one warp an output row
 * and two shared loads an FMA -> this: FP32 2^20, P = 64, 20 terms 18.4 -> 14.1; FP64 2^20, P = 32, 15 terms
 * 22.6 -> 14.4; FP64 2^17, P = 16, 24 terms 49 -> 29 (512 threads a block: the same, and 14 -> 23 at P = 256). */
constexpr int kCoarseMaxLevel = 6; /* M2M parents hold at most 2^6 boxes a plane */
constexpr int kCoarseStages = 2 * (kCoarseMaxLevel - 1) + 1, kCoarseThreads = 256;

template <class E> struct CoarseArgs {
  using R = typename E::R;
  R *phi, *psi;
  const R *m2m, *m2l, *top; /* TreeOps */
  long S1;                  /* planes / 2, all transforms of the execute */
  int T, Lm, Ll, resident, ns;
  TreeStage st[kCoarseStages];
};
/* Shared layout, in values: operators (all, or a buffer for one), phi levels 2 .. top, two levels of psi; the
 * stage table follows. */
template <class E> struct CoarseLay {
  int top, ph, ps[2], end;
  __host__ __device__ CoarseLay(int T, int Lm, int Ll, int resident) {
    const int Tq = tree_pitch(rows_kpad(T)), blk = tree_blk<E>(T);
    top = Lm >= 2 ? Lm + 1 : 2;
    if (Ll > top) top = Ll;
    ph = (resident ? 2 * (Lm - 1) + 1 + 8 * (Ll - 2) : Ll >= 3 ? 8 : 2) * blk;
    ps[0] = ph + ((2 << top) - 4) * Tq, ps[1] = ps[0] + (1 << Ll) * Tq, end = ps[1] + (Ll > 3 ? 1 << (Ll - 1) : 4) * Tq;
  }
};
template <class E> static size_t coarse_smem(int T, int Lm, int Ll, int resident) {
  return sizeof(typename E::R) * (size_t)CoarseLay<E>(T, Lm, Ll, resident).end + sizeof(TreeStage) * kCoarseStages;
}
template <class E> static void coarse_stages(CoarseArgs<E> &a) {
  const int T = a.T, Tp = rows_kpad(T), Tq = tree_pitch(Tp), blk = tree_blk<E>(T), nm = a.Lm - 1;
  const CoarseLay<E> lay(T, a.Lm, a.Ll, a.resident);
  auto phl = [&](int l) { return lay.ph + ((1 << l) - 4) * Tq; };
  auto psl = [&](int l) { return lay.ps[(a.Ll - l) & 1]; };
  a.ns = nm + 1 + a.Ll - 2;
  for (int i = 0; i < a.ns; ++i) {
    TreeStage g{};
    const int lM = a.Lm - i, lL = i - nm + 2; /* level of an M2M, of an M2L stage */
    g.op = !a.resident ? 0 : i < nm ? (lM - 2) * 2 * blk : i == nm ? nm * 2 * blk : (nm * 2 + 1 + (lL - 3) * 8) * blk;
    auto seg = [&](int base, int csh, int mul, int d0, int d1, int b0, int b1) {
      g.seg[g.nseg++] = TreeSeg{base, Tq, csh, mul, {d0, d1}, Tp, {g.op + b0 * blk, g.op + b1 * blk}};
    };
    g.npar = 1, g.ncol = Tp, g.gn = T, g.lv = 2;
    if (i < nm) {
      g.lv = lM, g.rows = 1 << lM, g.rsh = lM, g.so = phl(lM), g.nop = 2 * blk;
      seg(phl(lM + 1), lM + 1, 2, 0, 0, 0, 0), seg(phl(lM + 1), lM + 1, 2, 1, 1, 1, 1);
    } else if (i == nm) {
      g.rows = 4, g.rsh = 2, g.so = psl(2), g.nop = blk;
      seg(phl(2), 2, 1, 2, 2, 0, 0);
    } else {
      g.lv = lL, g.rows = 1 << (lL - 1), g.rsh = lL - 1, g.npar = 2, g.so = psl(lL), g.nop = 8 * blk;
      seg(psl(lL - 1), lL - 1, 1, 0, 0, 0, 4);
      seg(phl(lL), lL, 2, -2, -3, 1, 5), seg(phl(lL), lL, 2, 2, -2, 2, 6), seg(phl(lL), lL, 2, 3, 2, 3, 7);
    }
    const unsigned ncx = (unsigned)((sizeof(typename E::R) == 8 ? (g.ncol + 7) / 8 : (g.ncol + 3) / 4) * g.npar);
    g.rcp = ncx == 1 ? 0u : (unsigned)((0x100000000ull + ncx - 1) / ncx);
    a.st[i] = g;
  }
}

template <class E> __global__ void __launch_bounds__(kCoarseThreads) k_coarse(const __grid_constant__ CoarseArgs<E> a) {
  using R = typename E::R;
  extern __shared__ __align__(16) unsigned char tree_raw[];
  R *const sm = reinterpret_cast<R *>(tree_raw);
  const int T = a.T, Tp = rows_kpad(T), Tq = tree_pitch(Tp), blk = tree_blk<E>(T), nm = a.Lm - 1, ns = a.ns;
  const CoarseLay<E> lay(T, a.Lm, a.Ll, a.resident);
  TreeStage *const stages = reinterpret_cast<TreeStage *>(sm + lay.end);
  const long pl = blockIdx.x;
  auto stage_op = [&](int i) {
    const R *src = i < nm ? a.m2m + (long)(a.Lm - i - 2) * 2 * blk : i == nm ? a.top : a.m2l + (long)(i - nm - 1) * 8 * blk;
    tree_stage<R>(sm, src, a.st[i].nop);
  };
  tc::pdl_trigger();
  /* plan constants, before the wait for the kernel that made phi */
  if (a.resident) {
    tree_stage<R>(sm, a.m2m, nm * 2 * blk);
    tree_stage<R>(sm + nm * 2 * blk, a.top, blk);
    tree_stage<R>(sm + (nm * 2 + 1) * blk, a.m2l, (a.Ll - 2) * 8 * blk);
  } else {
    stage_op(0);
  }
  tree_commit();
  for (int e = threadIdx.x; e < ns * (int)(sizeof(TreeStage) / 4); e += kCoarseThreads)
    reinterpret_cast<int *>(stages)[e] = reinterpret_cast<const int *>(a.st)[e];
  tc::pdl_wait();
  for (int l = a.Lm >= 2 ? a.Lm + 1 : 2; l <= lay.top; ++l) { /* phi of the levels not made here */
    const R *src = a.phi + lvl_off(l, a.S1, T) + pl * (1L << l) * T;
    R *const dst = sm + lay.ph + ((1 << l) - 4) * Tq;
    for (int r = threadIdx.x >> 3; r < 1 << l; r += kCoarseThreads / 8)
      for (int c = threadIdx.x & 7; c < Tp; c += 8) dst[r * Tq + c] = c < T ? src[r * T + c] : R(0);
  }
  for (int i = 0; i < ns; ++i) {
    if (!a.resident && i > 0) {
      __syncthreads(); /* the stage before is done with the operator buffer */
      stage_op(i);
      tree_commit();
    }
    if (i == 0 || !a.resident) tree_wait<0>();
    __syncthreads(); /* this stage's operator and the stage before are in place */
    const TreeStage &sg = stages[i];
    R *const gbase = (i < nm ? a.phi : a.psi) + lvl_off(sg.lv, a.S1, T) + pl * (1L << sg.lv) * T;
    const int so = sg.so, gn = sg.gn, npar = sg.npar;
    blk_gemm(sm, sg, kCoarseThreads, [&](int r, int par, int c, R v0, R v1) {
      const int row = r * npar + par;
      tree_sput2<R>(sm + so + row * Tq + c, v0, v1);
      tree_put2<R>(gbase + (long)row * gn, gn, c, v0, v1);
    });
  }
}
