/*
 * FP64 row contractions of the FMM tree and leaf on the FP64 matrix instructions, sm_100a:
 * out[r][c] = sum_k A(r, k) B[k][c] over many rows r (section, re/im plane, box) with a small
 * operator B that a block keeps in shared memory in fragment order.
 *
 * Bound: the FP64 unit (37 TFLOP/s through either DFMA or mma.m8n8k4, both measured at 17 to 18
 * T fused multiply-adds/s) once nothing else is in its way.  A register-tiled DFMA kernel is not
 * bound by it: a 4 x 4 tile reads 8 values a lane from shared memory for 16 FMAs, twice what the
 * port delivers in the FMAs' time; the matrix instruction reads 2 values a lane for 8 FMAs a lane.
 * A warp takes whole tiles of rows and all of their columns.  Its A fragments come straight from
 * global memory into registers (8 rows x 32 contiguous bytes a load: whole sectors), so there is
 * no staging, no barrier after the operator is in place and nothing shared between warps.
 *
 * A problem (Rows*) names the row's source segments (each zero-padded to a multiple of 4 in K), which
 * of the NPAR operators a segment enters, and where a row's outputs go.
 */
#pragma once

/* Operator blocks of K rows and N columns (K padded to a multiple of 4, N to 8, zeros) as B
 * fragments of 4 x 8, one value a lane: lane (column % 8) * 4 + (k % 4). */
__host__ __device__ __forceinline__ int rows_kpad(int K) { return (K + 3) & ~3; }
__host__ __device__ __forceinline__ int rows_npad(int N) { return (N + 7) & ~7; }
__host__ __device__ __forceinline__ int rows_idx(int k, int c, int np) {
  return ((k >> 2) * (np >> 3) + (c >> 3)) * 32 + (c & 7) * 4 + (k & 3);
}
/* the (k, c) of element e of a block of np columns */
__device__ __forceinline__ void rows_kc(long e, int np, int &k, int &c) {
  const int lane = (int)(e & 31), q = (int)(e >> 5), nt = np >> 3;
  k = q / nt * 4 + (lane & 3), c = q % nt * 8 + (lane >> 2);
}
/* values of a T x T block, of the S2M operator (b x T) and of a section's leaf operator: the blocks of
 * psi (T x b) and of the boxes before, at and after (b x b) */
__host__ __device__ __forceinline__ int rows_blk(int T) { return rows_kpad(T) * rows_npad(T); }
__host__ __device__ __forceinline__ int rows_nleaf(int T, int b) { return (rows_kpad(T) + 3 * b) * rows_npad(b); }

/* ------------------------------------------------------------------------ problems */
/* Child level l, one row per parent box: the segments psi[B], phi[2B-2], phi[2B-1], phi[2B+2],
 * phi[2B+3]; operator 0 gives the left child (no phi[2B-1]), 1 the right child (no phi[2B+2]). */
struct RowsM2L {
  static constexpr int NSEG = 5, NPAR = 2, NP = 3;
  static constexpr bool kLeaf = false;
  const double *psi_par, *phi, *op;
  double *out;
  long rows;
  int T, lpar;
  static __device__ constexpr bool uses(int par, int seg) { return seg != (par ? 3 : 2); }
  static __device__ constexpr int blk(int par, int seg) { return par * 4 + (seg < 2 ? seg : par ? (seg == 2 ? 2 : 3) : seg - 1); }
  __device__ int len(int) const { return T; }
  __device__ void base(long r, int, const double *(&p)[NP]) const {
    const long pl = r >> lpar, B = r & ((1L << lpar) - 1), mask = (2L << lpar) - 1, b0 = pl << (lpar + 1);
    p[0] = psi_par + r * T;
    p[1] = phi + (b0 + ((2 * B - 2) & mask)) * T;
    p[2] = phi + (b0 + ((2 * B + 2) & mask)) * T;
  }
  static __device__ __forceinline__ const double *seg(const double *const (&p)[NP], int g, int T) {
    return g == 0 ? p[0] : g == 1 ? p[1] : g == 2 ? p[1] + T : g == 3 ? p[2] : p[2] + T;
  }
  __host__ __device__ int ncol() const { return T; }
  __device__ double *dst(long r, int par, int) const { return out + (2 * r + par) * T; }
};

/* Parent level: a row's children pair. */
struct RowsM2M {
  static constexpr int NSEG = 2, NPAR = 1, NP = 1;
  static constexpr bool kLeaf = false;
  const double *child, *op;
  double *out;
  long rows;
  int T;
  static __device__ constexpr bool uses(int, int) { return true; }
  static __device__ constexpr int blk(int, int seg) { return seg; }
  __device__ int len(int) const { return T; }
  __device__ void base(long r, int, const double *(&p)[NP]) const { p[0] = child + r * 2 * T; }
  static __device__ __forceinline__ const double *seg(const double *const (&p)[NP], int g, int T) { return p[0] + g * T; }
  __host__ __device__ int ncol() const { return T; }
  __device__ double *dst(long r, int, int) const { return out + r * T; }
};

/* Leaf multipoles: a row's b samples (batch z = transform). */
struct RowsS2M {
  static constexpr int NSEG = 1, NPAR = 1, NP = 1;
  static constexpr bool kLeaf = false;
  const double *xt, *op;
  double *out;
  long rows, M;
  int T, b, P;
  static __device__ constexpr bool uses(int, int) { return true; }
  static __device__ constexpr int blk(int, int) { return 0; }
  __device__ int len(int) const { return b; }
  __device__ void base(long r, int z, const double *(&p)[NP]) const { p[0] = xt + (2L * P * z + 2) * M + r * b; }
  static __device__ __forceinline__ const double *seg(const double *const (&p)[NP], int, int) { return p[0]; }
  __host__ __device__ int ncol() const { return T; }
  __device__ double *dst(long r, int, int z) const { return out + ((long)z * rows + r) * T; }
};

/* Leaf of section z + 1 (reference src/fmmfft.c:751-954): rows (transform, plane, box), segments
 * psi[box], x[box - 1], x[box + 1] and, its weights reach P / pi, last x[box].  For sc >= P/2 a box's first point lies in the box before
 * it (half-shifted): its value is that of the expansion and the window one box earlier with the
 * weights evalmh and cot[0 .. 3b), or for sc = P/2 the mean of both. */
struct RowsLeaf {
  static constexpr int NSEG = 4, NPAR = 1, NP = 4;
  static constexpr bool kLeaf = true;
  const double *psi_n, *xt, *op, *evalmh, *cot;
  double *u;
  long rows, M, s;
  int T, b, log2s, P;
  static __device__ constexpr bool uses(int, int) { return true; }
  __device__ int len(int seg) const { return seg == 0 ? T : b; }
  __device__ long plane(long r, int z) const { return (r >> (log2s + 1)) * 2 * (P - 1) + 2L * z + ((r >> log2s) & 1); }
  __device__ const double *xplane(long r, int z) const { return xt + (plane(r, z) + 2 * (r >> (log2s + 1)) + 2) * M; }
  /* the segments of row r shifted back by `back` boxes */
  __device__ void window(long r, int z, int back, const double *(&p)[NP]) const {
    const long bx = (r & (s - 1)) - back;
    const double *x = xplane(r, z);
    p[0] = psi_n + (plane(r, z) * s + (bx & (s - 1))) * T;
    p[1] = x + ((bx - 1) & (s - 1)) * b, p[2] = x + (bx & (s - 1)) * b, p[3] = x + ((bx + 1) & (s - 1)) * b;
  }
  __device__ void base(long r, int z, const double *(&p)[NP]) const { window(r, z, 0, p); }
  static __device__ __forceinline__ const double *seg(const double *const (&p)[NP], int g, int) { return p[g < 2 ? g : 5 - g]; }
  __host__ __device__ int ncol() const { return b; }
  __device__ double *dst(long r, int, int z) const { return u + plane(r, z) * M + (r & (s - 1)) * b; }
};

/* Two neighbouring columns of a row of n values (c even). */
__device__ __forceinline__ void rows_put2(double *row, int n, int c, double v0, double v1) {
  if ((n & 1) == 0) { /* the row starts on a pair: rows are n values apart */
    if (c < n) *reinterpret_cast<double2 *>(row + c) = make_double2(v0, v1);
  } else {
    if (c < n) row[c] = v0;
    if (c + 1 < n) row[c + 1] = v1;
  }
}

/* The half-shifted first points of the 8 rows r of a warp's lanes (4 lanes a row, lane t of a row
 * k = t, t + 4, ..), weights hw = evalmh (T, padded) and cot[0 .. 3b): the sum in every lane. */
__device__ __forceinline__ double rows_half_shift(const RowsLeaf &pb, long r, int z, const double *hw) {
  const int t = threadIdx.x & 3;
  const double *p[RowsLeaf::NP];
  pb.window(r, z, 1, p);
  double s = 0;
  for (int k = t; k < pb.T; k += 4) s = fma(p[0][k], hw[k], s);
#pragma unroll
  for (int g = 1; g < 4; ++g) {
    const double *w = hw + rows_kpad(pb.T) + (g - 1) * pb.b;
#pragma unroll 4
    for (int k = t; k < pb.b; k += 4) s = fma(p[g][k], w[k], s);
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s;
}

constexpr int kRowsThreads = 128;

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

/* RT tiles of 8 rows and NPAR x NT of 8 columns a warp; a block takes rows_blk rows of batch
 * blockIdx.y, with the nop values of that batch's operator in shared memory. */
template <class Prob, int NT, int RT>
__global__ void __launch_bounds__(kRowsThreads, 3) k_rows_f64(const __grid_constant__ Prob pb, long rows_blk, int nop) {
  extern __shared__ __align__(16) unsigned char rows_raw[];
  double *const sop = reinterpret_cast<double *>(rows_raw), *const hw = sop + nop;
  const int z = blockIdx.y, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  tc::pdl_trigger();
  { /* plan constants: staged before the wait for the kernel that made the rows */
    const double *op = pb.op + (long)(Prob::kLeaf ? z : 0) * nop;
    for (int e = 2 * threadIdx.x; e < nop; e += 2 * kRowsThreads) tc::cp_async16(tc::smem_addr(sop + e), op + e);
  }
  bool shifted = false;
  if constexpr (Prob::kLeaf) {
    shifted = 2 * (z + 1) >= pb.P;
    const int Tp = rows_kpad(pb.T);
    if (shifted)
      for (int e = threadIdx.x; e < Tp + 3 * pb.b; e += kRowsThreads)
        hw[e] = e < pb.T ? pb.evalmh[(long)z * pb.T + e] : e < Tp ? 0.0 : pb.cot[(long)z * 4 * pb.b + e - Tp];
  }
  tc::cp_async_wait_all();
  __syncthreads();
  tc::pdl_wait();
  const int ncol = pb.ncol(), nt = (ncol + 7) >> 3;
  const long rend0 = (blockIdx.x + 1) * rows_blk, rend = rend0 < pb.rows ? rend0 : pb.rows;
  for (long r0 = blockIdx.x * rows_blk + (threadIdx.x >> 5) * (8 * RT); r0 < rend; r0 += (kRowsThreads / 32) * 8 * RT) {
    const double *p[RT][Prob::NP];
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const long r = r0 + 8 * i + g;
      pb.base(r < pb.rows ? r : pb.rows - 1, z, p[i]);
    }
    for (int j0 = 0; j0 < nt; j0 += NT) { /* column groups (one but for wide leaves) */
      double acc[Prob::NPAR][RT][NT][2];
#pragma unroll
      for (int q = 0; q < Prob::NPAR; ++q)
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j) acc[q][i][j][0] = acc[q][i][j][1] = 0.0;
      int sofs = 0; /* leaf: the segment's block (the operator has them in box order) */
#pragma unroll
      for (int s = 0; s < Prob::NSEG; ++s) {
        const int len = pb.len(s), k4n = (len + 3) >> 2, bsz = k4n * nt * 32;
        const double *a[RT];
#pragma unroll
        for (int i = 0; i < RT; ++i) a[i] = Prob::seg(p[i], s, len) + t;
        const double *bq[Prob::NPAR];
#pragma unroll
        for (int q = 0; q < Prob::NPAR; ++q) {
          if constexpr (Prob::kLeaf) bq[q] = sop + sofs + (s == 2 ? bsz : s == 3 ? -bsz : 0) + j0 * 32 + lane;
          else bq[q] = sop + Prob::blk(q, s) * bsz + j0 * 32 + lane;
        }
        sofs += bsz;
#pragma unroll 4
        for (int k4 = 0; k4 < k4n; ++k4) {
          double av[RT];
#pragma unroll
          for (int i = 0; i < RT; ++i) av[i] = 4 * k4 + t < len ? __ldg(a[i] + 4 * k4) : 0.0;
#pragma unroll
          for (int q = 0; q < Prob::NPAR; ++q)
            if (Prob::uses(q, s))
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                const double bv = bq[q][(k4 * nt + j) * 32];
#pragma unroll
                for (int i = 0; i < RT; ++i) mma_f64(acc[q][i][j], av[i], bv);
              }
        }
      }
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const long r = r0 + 8 * i + g;
        if constexpr (Prob::kLeaf)
          if (shifted && j0 == 0) {
            const double h = rows_half_shift(pb, r < pb.rows ? r : pb.rows - 1, z, hw);
            if (t == 0) acc[0][i][0][0] = 2 * (z + 1) > pb.P ? h : 0.5 * (acc[0][i][0][0] + h);
          }
        if (r < rend)
#pragma unroll
          for (int q = 0; q < Prob::NPAR; ++q)
#pragma unroll
            for (int j = 0; j < NT; ++j)
              if (j0 + j < nt) rows_put2(pb.dst(r, q, z), ncol, 8 * (j0 + j) + 2 * t, acc[q][i][j][0], acc[q][i][j][1]);
      }
    }
  }
}
