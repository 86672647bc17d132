/*
 * tcgen05 leaf with both operands in shared memory, sm_100a: split-TF32 and BF16x3 plans, sections of 128
 * boxes up.  (BF16x3, 2^22, P = 64, 8 terms: 90 us in the BF16 warp-specialised form, 51 here.)
 *
 * D[r][0..N) = sum_k A(r, k) B[k][.] where the A of box r are its expansion psi[r] and the samples
 * x[r-1], x[r], x[r+1].  A tile is 128 consecutive boxes of one plane and keeps each box's data once,
 * split into TF32 hi and lo, in the MMA's core-matrix layout (8 rows x 16 bytes).  MMA row m = 8 g + j
 * is box 16 j + g, so the box before or after lies 8 rows away and a neighbour's segment of K is the
 * same shared data read from the row group before or after: a descriptor with another start address.
 * Groups -1 and 16 hold the tile's two halo boxes (and copies of the boxes of groups 15 and 0).  So a
 * value is loaded and split once a tile, where rows that carry their window do so three times, and N is
 * b + 1 columns, where the neighbour-sum form computes 3 b + 3.
 *
 * One CTA per SM, persistent over a contiguous run of tiles, roles in separate warps that hand work
 * over through mbarriers: 6 to 10 producer warps (global -> registers two tiles ahead, split, st.shared
 * into one of two stages), one thread that issues the MMAs (A_lo, then A_hi, against [B_hi; B_lo],
 * N = 2 npad, two accumulators in tensor memory) and copies the operators in, 4 epilogue warps.  A
 * producer lane holds one 16-byte chunk of a row; 8 lanes take the 8 rows of a group, 4 neighbouring
 * chunks a warp, so a warp instruction reads 8 x 64 contiguous bytes and its shared stores are free
 * of bank conflicts.
 *
 * Measured, neighbour-sum form -> this one (us a leaf): 2^20 P64 T20 31 -> 24, 2^22 P64 T8 66 -> 50,
 * 2^24 P64 T24 234 -> 197, 2^26 P256 T16 860 -> 648 (b = 32).  The small A_lo products enter the
 * accumulator while it is small: relative L2 error of the transform at 2^26 2.9e-7 -> 2.4e-7.  What bounds it:
 * 60% of a tile's 7 k cycles are the MMAs, about 130 cycles each where both operands (7 KB) come from
 * shared memory; the rest is producers and epilogue that share that memory's bandwidth with them.
 * M2M, S2M and M2L in this form were slower than rows of 16 lanes (2^24: 158 against 109, .., 286 / 217).
 *
 * Every wait is bounded (2 s); on expiry the CTA records kErrWaitTimeout, every role leaves its loop,
 * and the MMAs and copies in flight complete before tensor memory is freed.
 */
#pragma once

namespace tc {

constexpr int kSEpi = 4, kSMaxProd = 11; /* up to 16 warps: 4 a sub-partition, 128 registers a thread */
constexpr int kSMaxThreads = (kSMaxProd + kSEpi + 1) * 32;

/* A tile's A data and how K runs over it (in the problem, filled by the host). */
struct SsMap {
  int alen[2], acol[2];                  /* source arrays: floats of a row, first storage column (multiple of 8) */
  int nch;                               /* 16-byte chunks of a stored row */
  int nseg, scol[4], slen[4], sshift[4]; /* K segments: storage column, length (multiples of 8), box shift */
  int nst;                               /* stages: 2, or 1 where two do not fit */
  long s;                                /* rows of a strip (a power of two, a multiple of 128) */
};
constexpr int kSGroups = 18; /* row groups of a tile: 16 and the two of its halo boxes */
__host__ __device__ inline size_t ss_stage_bytes(int nch) { return (size_t)2 * kSGroups * nch * 128; }
__host__ __device__ inline size_t ss_b_bytes(int kpad, int npad) { return (size_t)2 * npad * kpad * 4; }
/* accumulator columns of a tile, and of the allocation (a power of two) */
__host__ __device__ inline int ss_acc_cols(int npad) { return 2 * npad <= 32 ? 32 : 2 * npad <= 64 ? 64 : 2 * npad <= 128 ? 128 : 256; }
/* rows staged by the epilogue: 128 of w floats, padded against bank conflicts */
__host__ __device__ inline size_t ss_out_bytes(int w) { return (size_t)kRows * (w + 4) * 4; }
__host__ __device__ inline size_t ss_smem_bytes(int kpad, int npad, int nch, int nst, int w) {
  return ss_b_bytes(kpad, npad) + nst * ss_stage_bytes(nch) + ss_out_bytes(w);
}
/* Producers: each warp keeps to one quad of chunks (a lane's source array and column are then fixed and
 * its addresses advance by constants) and takes every ss_split-th row group of it. */
__host__ __device__ inline int ss_quads(int nch) { return (nch + 3) >> 2; }
__host__ __device__ inline int ss_split(int nch) { /* warps a quad */
  const int q = ss_quads(nch);
  return q == 1 ? 8 : q == 2 ? 4 : q == 3 ? 3 : q <= 5 ? 2 : 1;
}
__host__ __device__ inline int ss_prod(int nch) { return ss_quads(nch) * ss_split(nch); }
__host__ __device__ inline int ss_steps(int nch) { return (kSGroups + ss_split(nch) - 1) / ss_split(nch); }

/* NSTEP >= ss_steps.  Prob: rows, batches, kpad, npad, bimg / bimg_stride (the operator of batch z as
 * the row form's image: hi rows then lo rows, core matrices), SsMap m, and
 *   const float *abase(int a, long r, int z)   row 0 of array a's strip that holds row r of batch z
 *   output rows of b floats go through shared memory (pitch b + 4): put_rows stores a warp's 32 of them in
 *   whole lines, adding what side_load took from global memory before the tile was ready; put_side(r, z, t)
 *   takes column b. */
template <class Prob, int NSTEP>
__global__ void __launch_bounds__(kSMaxThreads, 1) k_tc_ss(const __grid_constant__ Prob pb, int *status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ uint64_t full[2], empty[2], dfull[2], dempty[2], bbar, fin;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kpad = pb.kpad, npad = pb.npad, nch = pb.m.nch, nst = pb.m.nst;
  const uint32_t sbo = (uint32_t)nch * 128, half_bytes = (uint32_t)kSGroups * sbo; /* a stage's hi (or lo) part */
  const uint32_t b_bytes = (uint32_t)ss_b_bytes(kpad, npad), bsm = smem_addr(smem_raw);
  const uint32_t st0 = bsm + b_bytes, stage_bytes = 2 * half_bytes;
  const uint32_t ncols = 2u * ss_acc_cols(npad);
  const int nprod = ss_prod(nch), mma_warp = nprod + kSEpi;
  if (warp == mma_warp) tmem_alloc(&tmem_slot, ncols);
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full[i], nprod), mbar_init(&empty[i], 1);
      mbar_init(&dfull[i], 1), mbar_init(&dempty[i], kSEpi);
    }
    mbar_init(&bbar, 1);
    mbar_init(&fin, 1);
    fence_mbar_init();
    abort_flag = 0;
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const int tpb = (int)(pb.rows / kRows); /* tiles of a batch: whole strips of whole tiles */
  const int ntiles = tpb * pb.batches;
  const int tile0 = (int)(((long)ntiles * blockIdx.x) / gridDim.x), tile_end = (int)(((long)ntiles * (blockIdx.x + 1)) / gridDim.x);
  /* plan constants: the first operator is requested before the wait for the kernel that made A */
  pdl_trigger();
  if (warp == mma_warp && lane == 0 && tile0 < tile_end) {
    mbar_expect_tx(&bbar, b_bytes);
    bulk_g2s(bsm, pb.bimg + (long)(tile0 / tpb) * pb.bimg_stride, b_bytes, &bbar);
  }
  pdl_wait();

  if (warp < nprod) {
    /* ------------------------------------------------------------ producers */
    /* this lane: chunk c of row j8 of the groups g0, g0 + split, ..; array a, column cc of its rows */
    const int split = ss_split(nch), quad = warp / split, g0 = warp - quad * split;
    const int c = 4 * quad + (lane >> 3), j8 = lane & 7;
    const int a = 4 * c >= pb.m.acol[1] ? 1 : 0, cc = 4 * c - pb.m.acol[a];
    const int len = a ? pb.m.alen[1] : pb.m.alen[0];
    const bool stored = c < nch, data = stored && cc < len; /* a padding chunk holds zeros */
    const uint32_t soff = (uint32_t)g0 * sbo + (uint32_t)c * 128 + (uint32_t)j8 * 16, sstep = (uint32_t)split * sbo;
    const long pre = (long)(16 * j8 + g0 - 1) * len + cc, wrap = pb.m.s * len;
    const int pstep = split * len;
    /* lanes whose first / last row lies outside the tile (row -1, row 128): at a strip's end it wraps */
    const bool wfirst = g0 == 0 && j8 == 0;
    const int tlast = (kSGroups - 1 - g0) / split; /* this warp's last step */
    const bool has_end = j8 == 7 && g0 + tlast * split == kSGroups - 1;
    const long smask = pb.m.s - 1;
    float4 va[NSTEP], vb[NSTEP];
    auto load = [&](int tile, float4 (&v)[NSTEP]) {
      const int z = tile / tpb;
      const long r0 = (long)(tile - z * tpb) * kRows, box0 = r0 & smask;
      const float *p = pb.abase(a, r0, z) + box0 * len + pre;
      const bool first = wfirst && box0 == 0, last = has_end && box0 + kRows == pb.m.s;
#pragma unroll
      for (int t = 0; t < NSTEP; ++t) {
        const float *pt = p + t * pstep;
        if (t == 0 && first) pt += wrap;
        if (last && t == tlast) pt -= wrap;
        v[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (data && t <= tlast) v[t] = __ldg(reinterpret_cast<const float4 *>(pt));
      }
    };
    auto store = [&](int i, const float4 (&v)[NSTEP]) -> bool { /* tile number i of this CTA */
      const int st = nst == 2 ? i & 1 : 0, use = nst == 2 ? i >> 1 : i;
      bool ok = true;
      if (lane == 0) ok = t_wait(&empty[st], (uint32_t)((use & 1) ^ 1), &abort_flag, status);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) return false;
      const uint32_t base = st0 + (uint32_t)st * stage_bytes + soff;
#pragma unroll
      for (int t = 0; t < NSTEP; ++t)
        if (stored && t <= tlast) {
          const float x[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
          float h[4], l[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) h[q] = tf32_rna(x[q]), l[q] = tf32_rna(x[q] - h[q]);
          const uint32_t d = base + (uint32_t)t * sstep;
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" : : "r"(d), "f"(h[0]), "f"(h[1]), "f"(h[2]), "f"(h[3]) : "memory");
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" : : "r"(d + half_bytes), "f"(l[0]), "f"(l[1]), "f"(l[2]), "f"(l[3]) : "memory");
        }
      fence_smem_to_async(); /* each writer's stores, before the tensor core reads them */
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[st]);
      return true;
    };
    /* loads run two tiles ahead and are issued after a tile's fence, which waits for loads in flight */
    const int nt = tile_end - tile0;
    if (nt > 0) load(tile0, va);
    if (nt > 1) load(tile0 + 1, vb);
    for (int i = 0; i < nt; i += 2) {
      if (!store(i, va)) break;
      if (i + 2 < nt) load(tile0 + i + 2, va);
      if (i + 1 >= nt || !store(i + 1, vb)) break;
      if (i + 3 < nt) load(tile0 + i + 3, vb);
    }
  } else if (warp < mma_warp) {
    /* ------------------------------------------------------------ epilogue */
    const int q = warp & 3, m = 32 * q + lane, rel = 16 * (m & 7) + (m >> 3);
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    float *const outs = reinterpret_cast<float *>(smem_raw + b_bytes + nst * stage_bytes);
    for (int i = 0; i < tile_end - tile0; ++i) {
      const int tile = tile0 + i, z = tile / tpb, d = i & 1;
      const long r0 = (long)(tile - z * tpb) * kRows;
      /* staged rows: what their stores add is loaded before the wait for the tile's MMAs */
      typename Prob::Side side;
      pb.side_load(side, r0, z, q, lane);
      bool ok = true;
      if (lane == 0) ok = t_wait(&dfull[d], (uint32_t)((i >> 1) & 1), &abort_flag, status);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      fence_after_sync();
      const uint32_t acc = tmem + lane_addr + (uint32_t)d * (ncols >> 1);
      const long r = r0 + rel;
#pragma unroll 2
      for (int c0 = 0; c0 < npad; c0 += 8) {
        uint32_t th[8], tl[8];
        tmem_ld8_issue(acc + (uint32_t)c0, th);
        tmem_ld8_issue(acc + (uint32_t)(npad + c0), tl);
        tmem_ld_wait();
        reg_fence8(th);
        reg_fence8(tl);
        float t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = __uint_as_float(th[k]) + __uint_as_float(tl[k]);
        if (c0 < pb.b) {
          float *o = outs + m * (pb.b + 4) + c0;
          *reinterpret_cast<float4 *>(o) = make_float4(t[0], t[1], t[2], t[3]);
          *reinterpret_cast<float4 *>(o + 4) = make_float4(t[4], t[5], t[6], t[7]);
        } else if (c0 == pb.b) {
          pb.put_side(r, z, t[0]);
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dempty[d]);
      pb.put_rows(side, r0, z, q, lane, outs); /* this warp's 32 rows, whole rows a few at a time */
      __syncwarp();                            /* read before the next tile's rows are staged */
    }
  } else {
    if (lane == 0) {
      /* ---------------------------------------------------------- MMA issue, operators */
      const uint32_t idesc = make_idesc_tf32(2 * npad), b_sbo = (uint32_t)kpad * 32;
      int cur = tile0 < tile_end ? tile0 / tpb : -1;
      uint32_t bphase = 0;
      bool b_pending = tile0 < tile_end, ok = true;
      for (int i = 0; i < tile_end - tile0; ++i) {
        const int tile = tile0 + i, z = tile / tpb, d = i & 1, st = nst == 2 ? i & 1 : 0, use = nst == 2 ? i >> 1 : i;
        if (z != cur && pb.bimg_stride != 0) { /* the MMAs reading the old operator complete, then the new one comes */
          mma_commit(&bbar);
          ok = t_wait(&bbar, bphase, &abort_flag, status);
          bphase ^= 1;
          if (!ok) break;
          mbar_expect_tx(&bbar, b_bytes);
          bulk_g2s(bsm, pb.bimg + (long)z * pb.bimg_stride, b_bytes, &bbar);
          b_pending = true;
        }
        cur = z;
        if (b_pending) {
          ok = t_wait(&bbar, bphase, &abort_flag, status);
          if (!ok) break;
          bphase ^= 1, b_pending = false;
        }
        ok = t_wait(&dempty[d], (uint32_t)(((i >> 1) & 1) ^ 1), &abort_flag, status) &&
             t_wait(&full[st], (uint32_t)(use & 1), &abort_flag, status);
        if (!ok) break;
        fence_after_sync();
        const uint32_t dt = tmem + (uint32_t)d * (ncols >> 1);
        const uint32_t a0 = st0 + (uint32_t)st * stage_bytes;
        /* A_lo first, while the sums are small; descriptors advance by a K step of 256 bytes (16 units) */
        uint32_t on = 0; /* the first MMA overwrites the accumulator */
#pragma unroll 1
        for (int p = 1; p >= 0; --p) {
          uint64_t db = make_desc(bsm, 128, b_sbo);
#pragma unroll 1
          for (int g = 0; g < pb.m.nseg; ++g) {
            uint64_t da = make_desc(a0 + (uint32_t)p * half_bytes + (uint32_t)(1 + pb.m.sshift[g]) * sbo + (uint32_t)pb.m.scol[g] * 32, 128, sbo);
            const int ks = pb.m.slen[g] >> 3;
#pragma unroll 4
            for (int k = 0; k < ks; ++k, da += 16, db += 16) {
              mma_tf32(dt, da, db, idesc, on);
              on = 1;
            }
          }
        }
        mma_commit(&empty[st]);
        mma_commit(&dfull[d]);
      }
      /* every MMA and copy issued has completed before shared and tensor memory go */
      mma_commit(&fin);
      if (!t_wait_time(&fin, 0)) atomicExch(status, kErrWaitTimeout);
      if (b_pending) t_wait_time(&bbar, bphase);
    }
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (warp == mma_warp) tmem_dealloc(tmem, ncols);
}

}  // namespace tc
