// Flash attention (prefill) on the 5th-generation tensor cores.
//
// One CTA owns one or two tiles of 128 query rows of one head.  Both GEMMs of attention run as tcgen05.mma with
// accumulators in tensor memory:
//   S = Q . K^T   A = Q tile  [128 x HD]  (K-major, smem)   B = K tile [KVB x HD] (K-major, smem)   D = S in TMEM
//   O += P . V    A = P tile  [128 x KVB] (TMEM)            B = V tile [KVB x HD] (MN-major, smem)  D = O in TMEM
// Warp roles: warp 0 = TMA producer (K/V pages or rows through a ring), warp 1 = MMA issuer (and
// TMEM owner), then four softmax warps per tile: thread r owns query row r, which is TMEM lane r, so row max and
// row sum need no shuffles.  S is double buffered in TMEM: Q.K^T of block j+1 runs on the tensor core
// while the softmax warps work on block j, and P of block j lies in the columns that its S was read from.  The softmax warps
// never wait for P.V unless they have to rescale O.  The running maximum is only raised when a block exceeds
// it by more than 2^8 (the accumulator and the row sum share the stale maximum, so the final
// O / l is exact); raising it rescales the O accumulator in TMEM (tcgen05.ld / tcgen05.st).
//
// What bounds it: a block of one tile is a chain - S from TMEM, maximum, 64 exponentials a thread (512 cycles of the special-function
// unit for a warp), P back to TMEM - so that an SM needs two tiles in different places of their chains, and K/V
// must be under way earlier than that.  Two tiles in ONE CTA share the K/V blocks (half the copies, and they come in 2 KB boxes) and leave room for
// a ring of four; two CTAs of one tile each with two-block rings waited for their copies (2.1 us a block).  One tile to a CTA is for short
// inputs, where the CTAs would not fill the GPU otherwise, and for heads above 128.
// fp16, us (one tile with a two-block ring / now), heads of 128 unless said: 128 queries x 2048 keys 76 / 41 (the chain alone: one CTA per SM);
// 8192 causal, 32 + 8 heads 1324 / 890; 8192 queries on 16384 keys 3317 / 2462; 8 x 1024 causal 382 / 209; 6 x 1100, window 1024 194 / 104;
// 2 x 4096, heads of 64 588 / 417; 12 x 256 full 45 / 41 (one tile each); 93 causal, heads of 64 14.2 / 6.9.
// Then, with P in shared memory, a wait for P.V in every block and one lane in the MMA loop / as it is: 8192 causal 889 / 612; 7808 queries on 16000
// keys 2380 / 1593; 8 x 1024 causal 209 / 168; 2 x 4096, heads of 64 416 / 290; 6 x 1100, window 1024 104 / 83.  The copy loop run by its whole
// warp as well: 547; 1438; 157; 277; 80; 825 full, 8 + 1 heads of 256 43.6 / 32.5.
// A row's results stored 16 bytes at a time: 503; 1448; 114.5; 257; 67; 28.4; 12 x 256 full, heads of 80, behind a GEMM 26.9 / 20.2.
// V needs no transpose: the [tokens x 64] slabs a TMA box leaves in shared memory are exactly the
// MN-major 128-byte-swizzle operand layout.
//
// Same contract as the mma.sync kernel in attention.cu (varlen packed q, paged or contiguous KV,
// causal / window / boolean mask / segment ids, GQA).  Every wait is bounded.
#include "../common/dtype.cuh"
#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../rf_api.h"
#include "attn_params.cuh"

namespace rf {

constexpr int kFaRows = 128;          // query rows per CTA
constexpr int kFaBox = 16 * 128;      // one TMA box: 16 rows x 64 x 16-bit
constexpr int kFaMaxStages = 8;
constexpr float kFaRaise = 8.0f;      // raise the reference maximum only beyond 2^8

struct alignas(8) FaCtl {
  uint64_t q_full, kv_full[kFaMaxStages], kv_empty[kFaMaxStages], s_full[2][2], p_full[2][2], pv_done[2], o_full[2], settled;
  uint32_t tmem_base;
  int32_t abort_flag, issued;            // issued: K/V blocks that the producer has asked for
};

// HD: size of a query / key head, VD: of a value head, NQ: query tiles of a CTA.  Heads of 80 (vision towers' 72) arrive as two 64-column boxes
// whose second one runs into the next head or past the row's end (zeros); the products stop at 80.
template <int HD, int VD, int NQ> struct FaGeom {
  static constexpr int J = (HD + 63) / 64, JV = (VD + 63) / 64;      // 64-column chunks of the heads
  static constexpr int KVB = 64;                         // kv tokens per block
  static constexpr int kQTile = J * kFaRows * 128;
  static constexpr int kKBytes = J * KVB * 128;          // K of one stage, V behind it
  static constexpr int kStageBytes = kKBytes + JV * KVB * 128;
  static constexpr int kFixed = NQ * kQTile;             // the ring lies behind Q
  static constexpr int kSCols = NQ * 2 * KVB;            // S: two buffers per tile, then O per tile
  static constexpr int kOCols = (VD + 31) / 32 * 32;
  static constexpr int kTmemCols = kSCols + NQ * kOCols > 256 ? 512 : 256;
  static constexpr int kThreads = 64 + NQ * 128;
  static_assert(kSCols + NQ * kOCols <= 512, "accumulators do not fit tensor memory");
};
// bits a .. 63 set (all of them from a <= 0, none from a >= 64)
__device__ __forceinline__ uint64_t bits_from(int a) { return a >= 64 ? 0ull : ~0ull << max(a, 0); }
// 2^x on the special-function unit, results below 2^-126 flushed to zero
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T, int HD, int VD, int NQ>
__global__ void __launch_bounds__(FaGeom<HD, VD, NQ>::kThreads, NQ == 1 && HD <= 128 ? 2 : 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const AttnParams p, const int stages) {
  using G = FaGeom<HD, VD, NQ>;
  constexpr int J = G::J, JV = G::JV, KVB = G::KVB;
  // No alignment slack: two CTAs of the HD <= 128 configuration fill the SM's shared memory to within 2 KB.
  // The swizzled tiles need a 1024-byte aligned base, which the runtime provides when the kernel has no
  // static shared memory; a misaligned base is reported instead of being used.
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) report_status(p.status, kStatusBadArgument, kTagAttnPrefill, (int)(smem_u32(smem_raw) & 1023u));
    return;
  }
  uint8_t* qsm = smem;
  uint8_t* kvsm = smem + G::kFixed;
  FaCtl* ctl = reinterpret_cast<FaCtl*>(kvsm + (size_t)stages * G::kStageBytes);

  // heads run fastest, the last rows of a sequence first: under a causal mask they have the most keys, and what is left for the end is short
  const int h = blockIdx.x, seq = blockIdx.z;
  const int qt0 = (int)(gridDim.y - 1 - blockIdx.y) * NQ;   // first query tile of this CTA
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int qlen = p.q_len[seq];
  if (qt0 * kFaRows >= qlen) return;                      // before any barrier or allocation
  const int kvlen = p.kv_len[seq];
  const int kvh = h / p.G;
  const int pt_row = p.slot ? p.slot[seq] : seq;
  const int qpos0 = kvlen - qlen;                         // position of query row 0 on the kv axis
  const int q_row0 = p.q_start[seq] + qt0 * kFaRows;
  const int tiles = NQ == 1 ? 1 : min(NQ, (qlen - qt0 * kFaRows + kFaRows - 1) / kFaRows);   // tiles that have rows
  const int first = qpos0 + qt0 * kFaRows;                // position of the CTA's first query row
  int kv_lo = 0;
  if (p.window > 0) kv_lo = max(0, first - p.window + 1);
  if (p.chunk > 0) kv_lo = max(kv_lo, first / p.chunk * p.chunk);   // the first row's chunk
  kv_lo &= ~(KVB - 1);
  // blocks of the kept first positions come first, then those from the first row's window or chunk on
  const int keep_blk = min((p.keep_first + KVB - 1) / KVB, kv_lo / KVB);
  auto block_start = [&](int j) { return j < keep_blk ? j * KVB : kv_lo + (j - keep_blk) * KVB; };
  // a tile's blocks: up to the last key its last row sees (the CTA's tiles walk the same list, the first one may stop earlier)
  auto blocks_of = [&](int t) {
    const int rows = min(kFaRows, qlen - (qt0 + t) * kFaRows);
    const int hi = p.causal ? min(kvlen, first + t * kFaRows + rows) : kvlen;
    return hi > kv_lo ? keep_blk + (hi - kv_lo + KVB - 1) / KVB : 0;
  };
  int nblk_t[NQ];
#pragma unroll
  for (int t = 0; t < NQ; ++t) nblk_t[t] = t < tiles ? blocks_of(t) : 0;
  const int nblk = NQ == 1 ? nblk_t[0] : max(nblk_t[0], nblk_t[NQ - 1]);

  if (tid == 0) {
    mbar_init(&ctl->q_full, 1);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctl->kv_full[s], 1);
      mbar_init(&ctl->kv_empty[s], 1);
    }
    for (int t = 0; t < NQ; ++t) {
      for (int b = 0; b < 2; ++b) {
        mbar_init(&ctl->s_full[t][b], 1);
        mbar_init(&ctl->p_full[t][b], 4);              // per buffer: a warp may be a block ahead of its tile's others
      }
      mbar_init(&ctl->pv_done[t], 1);
      mbar_init(&ctl->o_full[t], 1);
    }
    mbar_init(&ctl->settled, 1);
    ctl->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, (uint32_t)G::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  pdl_launch_dependents();     // only after this CTA owns its TMEM columns
  pdl_wait();                  // q, k, v come from the previous kernel
  volatile int32_t* abort_flag = &ctl->abort_flag;
  uint64_t limit = kLocalWaitNs;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer ----
    // the warp reads 32 page numbers at a time, one elected lane issues the copies
    constexpr int kPagesPerBlock = KVB / 16, kBlocksPerFetch = 32 / kPagesPerBlock;
    const bool lead = elect_one();
    if (lead && nblk > 0) {                                 // nobody would wait for it without keys
      mbar_arrive_expect_tx(&ctl->q_full, (uint32_t)(tiles * G::kQTile));
      for (int t = 0; t < tiles; ++t)
#pragma unroll
        for (int c = 0; c < J; ++c)
          tma_load_2d(qsm + t * G::kQTile + c * (kFaRows * 128), &tmQ, &ctl->q_full, h * HD + c * 64, q_row0 + t * kFaRows);
    }
    const int row0 = p.paged ? 0 : p.kv_start[seq];
    int pages = 0, s = 0;
    uint32_t phase = 1;                                     // nothing is waited for on the first turn of the ring
    int j = 0;
    for (; j < nblk; ++j) {
      if (p.paged && j % kBlocksPerFetch == 0)
        pages = p.page_table[(size_t)pt_row * p.pt_stride + min(block_start(j + lane / kPagesPerBlock) / 16 + lane % kPagesPerBlock, p.pt_stride - 1)];
      int block_pages[kPagesPerBlock];
#pragma unroll
      for (int w = 0; w < kPagesPerBlock; ++w) block_pages[w] = __shfl_sync(0xffffffffu, pages, (j % kBlocksPerFetch) * kPagesPerBlock + w);
      const bool free = role_wait(&ctl->kv_empty[s], phase, &limit, &ctl->abort_flag, p.status, kStatusTmaTimeout, kTagAttnPrefill, j, 32);
      if (free && lead) {
        uint8_t* ks = kvsm + s * G::kStageBytes;
        uint8_t* vs = ks + G::kKBytes;
        mbar_arrive_expect_tx(&ctl->kv_full[s], (uint32_t)G::kStageBytes);
        // Whole blocks are always loaded: rows past the sequence end are other (finite) cache rows or the
        // zero fill beyond the tensor, and their probabilities are forced to zero.
        if (p.paged) {
#pragma unroll
          for (int w = 0; w < kPagesPerBlock; ++w) {
            const int row = (block_pages[w] * p.Hkv + kvh) * 16;
#pragma unroll
            for (int c = 0; c < J; ++c) {
              tma_load_2d(ks + c * (KVB * 128) + w * kFaBox, &tmK, &ctl->kv_full[s], c * 64, row);
              if (c < JV) tma_load_2d(vs + c * (KVB * 128) + w * kFaBox, &tmV, &ctl->kv_full[s], c * 64, row);
            }
          }
        } else {
          const int row = row0 + block_start(j);
#pragma unroll
          for (int c = 0; c < J; ++c) {
            tma_load_2d(ks + c * (KVB * 128), &tmK, &ctl->kv_full[s], kvh * HD + c * 64, row);
            if (c < JV) tma_load_2d(vs + c * (KVB * 128), &tmV, &ctl->kv_full[s], kvh * VD + c * 64, row);
          }
        }
      }
      if (!agreed(free)) break;
      if (++s == stages) { s = 0; phase ^= 1u; }
    }
    if (lead) ctl->issued = j;
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer ----
    if (nblk > 0) {
      const bool lead = elect_one();
      const uint32_t idesc_qk = umma_idesc_f16(kFaRows, KVB, Num<T>::kFmt, 0);
      const uint32_t idesc_pv = umma_idesc_f16(kFaRows, VD, Num<T>::kFmt, 1);
      // One lane issues every MMA, twelve per tile and block: the operand descriptors are made once and advance by constants (16-byte units)
      const uint64_t q_desc = umma_desc_k128(smem_u32(qsm));
      const uint64_t k_desc0 = umma_desc_k128(smem_u32(kvsm)), v_desc0 = umma_desc_mn128(smem_u32(kvsm) + G::kKBytes, (uint32_t)(KVB * 128));
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        role_wait(bar, parity, &limit, &ctl->abort_flag, p.status, kStatusMmaTimeout, kTagAttnPrefill, 1000);
      };
      wait(&ctl->q_full, 0);
      auto issue_qk = [&](int t, int j, int s, uint32_t ph) {
        const int b = j & 1;
        wait(&ctl->kv_full[s], ph);
        // this S buffer holds P of block j - 2 until its product is done (the other tile's products are in the queue behind that one)
        if (j >= 2) wait(&ctl->pv_done[t], (uint32_t)j & 1u);
        tc_fence_after_sync();
        if (lead) {
          const uint64_t qd = q_desc + (uint32_t)(t * (G::kQTile >> 4)), kd = k_desc0 + (uint32_t)(s * (G::kStageBytes >> 4));
          const uint32_t d = tmem_base + (uint32_t)((t * 2 + b) * KVB);
#pragma unroll
          for (int c = 0; c < J; ++c)
#pragma unroll
            for (int kk = 0; kk < 4 && c * 64 + kk * 16 < HD; ++kk)
              umma_f16(d, qd + (uint32_t)((c * kFaRows * 128 + kk * 32) >> 4), kd + (uint32_t)((c * KVB * 128 + kk * 32) >> 4), idesc_qk, (c | kk) ? 1u : 0u);
          umma_commit(&ctl->s_full[t][b]);
        }
      };
#pragma unroll
      for (int t = 0; t < NQ; ++t)
        if (nblk_t[t] > 0) issue_qk(t, 0, 0, 0);
      int s = 0, s_next = 1;                                          // stages of blocks j and j + 1 (at least two), phase of the latter
      uint32_t ph_next = 0;
      for (int j = 0; j < nblk; ++j) {
#pragma unroll
        for (int t = 0; t < NQ; ++t)
          if (j + 1 < nblk_t[t]) issue_qk(t, j + 1, s_next, ph_next);      // runs while the softmax warps work on block j
        const uint64_t vd = v_desc0 + (uint32_t)(s * (G::kStageBytes >> 4));
#pragma unroll
        for (int t = 0; t < NQ; ++t) {
          if (j >= nblk_t[t]) continue;
          wait(&ctl->p_full[t][j & 1], (uint32_t)(j >> 1) & 1u);
          tc_fence_after_sync();
          if (lead) {
#pragma unroll
            for (int k = 0; k < KVB / 16; ++k)
              umma_f16_ts(tmem_base + (uint32_t)(G::kSCols + t * G::kOCols), tmem_base + (uint32_t)((t * 2 + (j & 1)) * KVB + k * 8),
                          vd + (uint32_t)((k * kFaBox) >> 4), idesc_pv, (j | k) ? 1u : 0u);
            umma_commit(&ctl->pv_done[t]);
            if (j + 1 == nblk_t[t]) umma_commit(&ctl->o_full[t]);
          }
        }
        if (lead && limit) umma_commit(&ctl->kv_empty[s]);            // every tile's products with this block
        s = s_next;
        if (++s_next == stages) { s_next = 0; ph_next ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------- softmax / correction / epilogue ----
    const int t = NQ == 1 ? 0 : (warp - 2) >> 2;          // this warp's query tile
    const int nblk = t == 0 ? nblk_t[0] : nblk_t[NQ - 1];
    const int quarter = warp & 3;                         // TMEM lanes this warp may touch
    const int r = quarter * 32 + lane;                    // query row of this thread inside the tile
    const int qi = (qt0 + t) * kFaRows + r;               // row index inside the sequence
    const uint32_t o_col = (uint32_t)(G::kSCols + t * G::kOCols);
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint8_t* mrow = p.mask ? p.mask + (size_t)seq * p.mask_seq_stride + (size_t)min(qi, qlen - 1) * p.mask_ld : nullptr;
    const int sq = (p.seg_q && qi < qlen) ? p.seg_q[p.q_start[seq] + qi] : 0;
    const int kv0 = p.paged ? 0 : p.kv_start[seq];
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    // bounds of the valid kv positions of this row that do not depend on data: [lo, hi]
    const int hi_row = min(kvlen - 1, p.causal ? qpos0 + qi : 0x7fffffff);
    int lo_row = p.window > 0 ? qpos0 + qi - p.window + 1 : 0;
    if (p.chunk > 0) lo_row = max(lo_row, (qpos0 + qi) / p.chunk * p.chunk);
    const bool data_mask = mrow != nullptr || p.seg_q != nullptr;
    const float fall = p.slopes ? p.slopes[h] * (p.rates ? 1.f : kLog2e) : 0.f, rate = p.rates ? p.rates[h] : 0.f;
    const float score_mul = p.slopes ? 1.f : p.scale_log2;
    for (int j = 0; j < nblk; ++j) {
      const int b = j & 1;
      const bool have = role_wait(&ctl->s_full[t][b], (uint32_t)(j >> 1) & 1u, &limit, &ctl->abort_flag, p.status, kStatusEpilogueTimeout, kTagAttnPrefill, r);
      if (!have || *abort_flag) { ok = false; break; }
      tc_fence_after_sync();
      const int t0 = block_start(j);
      const uint32_t s_addr = lane_base + (uint32_t)((t * 2 + b) * KVB);
      // the whole row of S for this block: all loads in flight, one wait
      uint32_t sv[KVB];
#pragma unroll
      for (int c0 = 0; c0 < KVB; c0 += 32) tmem_ld32(s_addr + c0, *reinterpret_cast<uint32_t(*)[32]>(&sv[c0]));
      tmem_ld_wait();
      // masking: interior blocks need none; edge blocks compare against the row's [lo, hi]; boolean
      // masks and segment ids (rare) take the per-element path
      const bool edge = __any_sync(0xffffffffu, (t0 < lo_row && t0 + KVB > p.keep_first) || t0 + KVB - 1 > hi_row) || data_mask;
      if (p.rates) {                                        // finished scores: scaled, less the fall over the distance's logarithm
        const float back = (float)(qpos0 + qi - t0);
#pragma unroll
        for (int i = 0; i < KVB; ++i)
          sv[i] = __float_as_uint(fmaf(-fall, log2_distance(rate, back - (float)i), __uint_as_float(sv[i]) * p.scale_log2));
      } else if (p.slopes) {                                // ... or over the distance
        const float past = (float)(t0 - qpos0 - qi);
#pragma unroll
        for (int i = 0; i < KVB; ++i)
          sv[i] = __float_as_uint(fmaf(fall, past + (float)i, __uint_as_float(sv[i]) * p.scale_log2));
      }
      // Inside the mask the scores stay as they came and `mul` goes into the exponent's multiply-add; elsewhere they are finished here.
      // Four running maxima (and sums below): one would be a chain of 64 dependent instructions.
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, mul = 1.f;
      if (!edge && score_mul > 0.f) {
        mul = score_mul;
#pragma unroll
        for (int i = 0; i < KVB; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[i]));
#pragma unroll
        for (int i = 0; i < 4; ++i) mx4[i] *= score_mul;
      } else if (!data_mask && score_mul > 0.f) {
        // a block on the diagonal or on the edge of a window: the row's keys as one bit each.  The general loop below, with its tests for data masks
        // behind every key, took some 3 us a block (128 x 128 causal, 32 + 8 heads of 128: 17.1 us, 10.4 with this), and a causal tile has two such blocks.
        mul = score_mul;
        const uint64_t bits = (bits_from(lo_row - t0) | ~bits_from(p.keep_first - t0)) & ~bits_from(hi_row - t0 + 1);
        const uint32_t w32[2] = {(uint32_t)bits, (uint32_t)(bits >> 32)};
#pragma unroll
        for (int i = 0; i < KVB; ++i) {
          const float x = (w32[i >> 5] & (1u << (i & 31))) ? __uint_as_float(sv[i]) : -INFINITY;
          sv[i] = __float_as_uint(x);
          mx4[i & 3] = fmaxf(mx4[i & 3], x);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) mx4[i] *= score_mul;
      } else if (!edge) {
#pragma unroll
        for (int i = 0; i < KVB; ++i) {
          const float v = __uint_as_float(sv[i]) * score_mul;
          sv[i] = __float_as_uint(v);
          mx4[i & 3] = fmaxf(mx4[i & 3], v);
        }
      } else if (mrow != nullptr && p.seg_q == nullptr && ((reinterpret_cast<uintptr_t>(mrow) + (uintptr_t)t0) & 15u) == 0 &&
                 t0 + KVB <= p.mask_ld) {
        // boolean mask, 16-byte aligned and wholly inside the row: the block's KVB mask bytes come as 16-byte
        // loads that are all in flight at once (byte loads chained behind the range test cost a cache round
        // trip each and made a 31 x 331 problem take 60 us)
        uint4 mv[KVB / 16];
        const uint4* m16 = reinterpret_cast<const uint4*>(mrow + t0);
#pragma unroll
        for (int c = 0; c < KVB / 16; ++c) mv[c] = __ldg(m16 + c);
#pragma unroll
        for (int i = 0; i < KVB; ++i) {
          const int tk = t0 + i;
          const uint32_t word = reinterpret_cast<const uint32_t*>(&mv[i >> 4])[(i >> 2) & 3];
          const bool v = tk >= lo_row && tk <= hi_row && ((word >> ((i & 3) * 8)) & 0xffu) != 0;
          const float x = v ? __uint_as_float(sv[i]) * score_mul : -INFINITY;
          sv[i] = __float_as_uint(x);
          mx4[i & 3] = fmaxf(mx4[i & 3], x);
        }
      } else if (mrow == nullptr && p.seg_q != nullptr) {
        // segment ids alone: a lane fetches those of two keys and the warp hands them round (a load behind every key's range test: 1 x 1024 rows,
        // 16 + 4 heads of 64, 153 us, 30.4 so)
        int sk[KVB / 32];
#pragma unroll
        for (int c = 0; c < KVB / 32; ++c) {
          const int tk = t0 + c * 32 + lane;
          sk[c] = tk < kvlen ? p.seg_k[kv0 + tk] : 0;
        }
        const uint64_t bits = bits_from(lo_row - t0) & ~bits_from(hi_row - t0 + 1);
        const uint32_t w32[2] = {(uint32_t)bits, (uint32_t)(bits >> 32)};
#pragma unroll
        for (int i = 0; i < KVB; ++i) {
          const bool same = __shfl_sync(0xffffffffu, sk[i >> 5], i & 31) == sq;
          const float x = same && (w32[i >> 5] & (1u << (i & 31))) ? __uint_as_float(sv[i]) * score_mul : -INFINITY;
          sv[i] = __float_as_uint(x);
          mx4[i & 3] = fmaxf(mx4[i & 3], x);
        }
      } else {
#pragma unroll
        for (int i = 0; i < KVB; ++i) {
          const int tk = t0 + i;
          bool v = (tk >= lo_row || tk < p.keep_first) && tk <= hi_row;
          if (data_mask && v) {
            if (mrow) v = mrow[tk] != 0;
            if (p.seg_q && v) v = p.seg_k[kv0 + tk] == sq;
          }
          const float x = v ? __uint_as_float(sv[i]) * score_mul : -INFINITY;
          sv[i] = __float_as_uint(x);
          mx4[i & 3] = fmaxf(mx4[i & 3], x);
        }
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const bool raise = mx > m_ref + kFaRaise || (m_ref == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, raise)) {               // tcgen05.ld/st are warp-wide
        const float m_new = raise ? mx : m_ref;
        const float alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - m_new);
        if (j > 0) {
          // O belongs to the tensor core until P.V of the previous block has finished (that of the block before is: it was issued ahead of
          // this block's Q.K^T, so the parity is not ambiguous)
          ok = role_wait(&ctl->pv_done[t], (uint32_t)(j - 1) & 1u, &limit, &ctl->abort_flag, p.status, kStatusEpilogueTimeout, kTagAttnPrefill, r);
          if (!ok) break;
          tc_fence_after_sync();
#pragma unroll 1
          for (int c0 = 0; c0 < VD; c0 += 32) {
            uint32_t ov[32];
            tmem_ld32(lane_base + o_col + (uint32_t)c0, ov);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * (raise ? alpha : 1.f));
            tmem_st32(lane_base + o_col + (uint32_t)c0, ov);
          }
          tmem_st_wait();
        }
        if (raise) {
          l *= alpha;
          m_ref = m_new;
        }
      }
      // probabilities against the reference maximum -> 16-bit P in place of the first half of S, two keys to a column
      const float mref = m_ref == -INFINITY ? 0.f : m_ref;
      float rs[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[KVB / 2];
#pragma unroll
      for (int i = 0; i < KVB / 2; ++i) {
        const float e0 = ex2(fmaf(__uint_as_float(sv[2 * i]), mul, -mref));         // masked entries are -inf -> 0
        const float e1 = ex2(fmaf(__uint_as_float(sv[2 * i + 1]), mul, -mref));
        rs[(2 * i) & 3] += e0;
        rs[(2 * i + 1) & 3] += e1;
        const typename Num<T>::T2 v = Num<T>::from_f2(e0, e1);
        pk[i] = *reinterpret_cast<const uint32_t*>(&v);
      }
      tmem_st32(s_addr, pk);
      l += (rs[0] + rs[1]) + (rs[2] + rs[3]);
      tmem_st_wait();
      // P (and a rescaled O) are ready for the tensor core
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->p_full[t][b]);
    }
    // epilogue: O / l
    if (nblk > 0) ok &= role_wait(&ctl->o_full[t], 0, &limit, &ctl->abort_flag, p.status, kStatusEpilogueTimeout, kTagAttnPrefill, r);
    ok = agreed(ok && !*abort_flag);
    tc_fence_after_sync();
    if (ok) {
      if (p.sink && l > 0.f) l += exp2f(p.sink[h] * kLog2e - m_ref);
      float inv = l > 0.f ? 1.f / l : 0.f;
      const T* grow = p.gate ? reinterpret_cast<const T*>(p.gate) + (size_t)(p.q_start[seq] + qi) * p.ld_gate + (p.gate_by_head ? h : h * VD) : nullptr;
      if (p.gate_by_head && grow && qi < qlen) {
        inv *= sigmoid_fast(Num<T>::to_f(grow[0]));
        grow = nullptr;
      }
      T* orow = reinterpret_cast<T*>(p.out) + (size_t)(p.q_start[seq] + qi) * p.ldo + (size_t)h * VD;
#pragma unroll 1
      for (int c0 = 0; c0 < VD; c0 += 32) {
        uint32_t ov[32];
        if (nblk > 0) {
          tmem_ld32(lane_base + o_col + (uint32_t)c0, ov);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = 0u;
        }
        if (qi < qlen) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (c0 + u * 8 >= VD) break;
            float f8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f8[i] = __uint_as_float(ov[u * 8 + i]) * inv;
            if (grow) {
              float g8[8];
              load8(grow + c0 + u * 8, g8);
#pragma unroll
              for (int i = 0; i < 8; ++i) f8[i] *= sigmoid_fast(g8[i]);
            }
            store8(orow + c0 + u * 8, f8);
          }
        }
      }
    }
  }
  // ----------------------------------------------------------------- teardown ----
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {           // a role gave up: what the others had started ends first
    if (warp == 0) {
      mbar_wait(&ctl->q_full, 0, kSettleNs);
      settle_copies(ctl->kv_full, stages, ctl->issued);
    }
    if (warp == 1) settle_mmas(&ctl->settled);
  }
  if (warp == 1) tmem_dealloc(tmem_base, (uint32_t)G::kTmemCols);
}

template <typename T, int HD, int VD, int NQ>
static int launch_prefill_tc_n(const RfAttn* a, const AttnParams& p, cudaStream_t s) {
  using G = FaGeom<HD, VD, NQ>;
  CUtensorMap tmQ, tmK, tmV;
  int rc;
  if (a->k_pool) {
    const uint64_t rows = (uint64_t)a->pool_pages * a->Hkv * 16;
    rc = make_tmap_2d(&tmK, a->k_pool, a->dtype, 2, a->hd, rows, a->hd, 64, 16, true);
    if (rc) return rc;
    rc = make_tmap_2d(&tmV, a->v_pool, a->dtype, 2, a->hd, rows, a->hd, 64, 16, true);
  } else {
    rc = make_tmap_2d(&tmK, a->k, a->dtype, 2, (uint64_t)a->Hkv * a->hd, a->kv_rows_total, a->ldk, 64, G::KVB, true);
    if (rc) return rc;
    rc = make_tmap_2d(&tmV, a->v, a->dtype, 2, (uint64_t)a->Hkv * VD, a->kv_rows_total, a->ldv, 64, G::KVB, true);
  }
  if (rc) return rc;
  rc = make_tmap_2d(&tmQ, a->q, a->dtype, 2, (uint64_t)a->Hq * a->hd, a->q_rows_total, a->ldq, 64, kFaRows, true);
  if (rc) return rc;
  dim3 grid(a->Hq, ceil_div(a->max_q_len, kFaRows * NQ), a->num_seqs);
  RF_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "prefill attention: %u row tiles of %u sequences", grid.y, grid.z);
  // One-tile CTAs of heads up to 128 sit two to an SM with a ring of two blocks once there are more of them than SMs; a CTA that has its SM to
  // itself takes what shared memory there is.
  const bool pair = NQ == 1 && HD <= 128 && (long)grid.x * grid.y * grid.z > sm_count();
  const int room = (pair ? 113 : 226) * 1024 - G::kFixed - (int)sizeof(FaCtl);
  const int stages = std::min(kFaMaxStages, room / G::kStageBytes);
  RF_REQUIRE(stages >= 2, "prefill attention: heads of %d / %d do not fit shared memory", HD, VD);
  const size_t smem = (size_t)G::kFixed + (size_t)stages * G::kStageBytes + sizeof(FaCtl);
  auto kfn = attn_prefill_tc_kernel<T, HD, VD, NQ>;
  RF_ALLOW_SMEM_PER_DEVICE(kfn, 227 * 1024);
  RF_CUDA_CHECK(::rf::launch_k(kfn, grid, dim3(G::kThreads), smem, s, 1, tmQ, tmK, tmV, p, stages));
  ::rf::count_launch();
  return RF_OK;
}

template <typename T, int HD, int VD = HD>
static int launch_prefill_tc_t(const RfAttn* a, const AttnParams& p, cudaStream_t s) {
  if constexpr (HD <= 128) {
    // Two tiles to a CTA where that still makes about one CTA per SM and the tiles have more than a few blocks to share (12 x 256 rows and keys,
    // 16 heads of 128: 47 us with two tiles, 42 with one).  Not under masks by data, whose blocks are bound by the tests behind every score: there
    // two CTAs of one tile hide each other's loads of the mask, and a sequence's odd last tile does not leave half an SM idle (12 x 300, 16 + 4
    // heads of 64, boolean mask: 53.6 us with two tiles, 39.2 with one).
    if (!a->mask && !a->seg_q && a->max_q_len > 2 * kFaRows && 4l * ceil_div(a->max_q_len, 2 * kFaRows) * a->Hq * a->num_seqs >= 3l * sm_count())
      return launch_prefill_tc_n<T, HD, VD, 2>(a, p, s);
  }
  return launch_prefill_tc_n<T, HD, VD, 1>(a, p, s);
}

// Entry used by rf_attn_prefill (attention.cu): `p` is already filled from `a`.
int launch_prefill_tc(const RfAttn* a, const AttnParams& p, cudaStream_t s) {
  RF_REQUIRE(a->q_start && a->q_len && a->max_q_len > 0 && a->q_rows_total > 0,
             "prefill attention needs q_start, q_len, max_q_len, q_rows_total");
  if (a->dtype == 0) {
    if (a->hd == 64) return launch_prefill_tc_t<__half, 64>(a, p, s);
    if (a->hd == 80) return launch_prefill_tc_t<__half, 80>(a, p, s);
    if (a->hd == 128) return launch_prefill_tc_t<__half, 128>(a, p, s);
    if (a->hd == 192) return launch_prefill_tc_t<__half, 192, 128>(a, p, s);
    return launch_prefill_tc_t<__half, 256>(a, p, s);
  }
  if (a->hd == 64) return launch_prefill_tc_t<__nv_bfloat16, 64>(a, p, s);
  if (a->hd == 80) return launch_prefill_tc_t<__nv_bfloat16, 80>(a, p, s);
  if (a->hd == 128) return launch_prefill_tc_t<__nv_bfloat16, 128>(a, p, s);
  if (a->hd == 192) return launch_prefill_tc_t<__nv_bfloat16, 192, 128>(a, p, s);
  return launch_prefill_tc_t<__nv_bfloat16, 256>(a, p, s);
}

}  // namespace rf
