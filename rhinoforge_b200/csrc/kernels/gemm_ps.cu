// Persistent tcgen05 GEMM for large token counts (prefill):  out[M,N] = epilogue( x[M,K] . w[N,K]^T ).
//
// One CTA per SM walks a list of (128*MT) x BN output tiles.  Three roles run concurrently:
//   warp 0      TMA producer: the activation tile(s) by tensor map, the weight blocks (tile-major layout) by
//               bulk copy; its ring runs ahead into the next tile while the current one is still multiplying;
//   warp 1      MMA issuer: accumulates a tile into an accumulator buffer in tensor memory;
//   warps 2..   epilogue (four warps per 128-row half): scale, bias, activation / GLU, residual, store.
// MT = 1: 128 x BN tiles and TWO accumulator buffers, so a tile's epilogue runs under the next tile's MMAs.
// MT = 2: 256 x BN tiles; each weight tile in shared memory feeds two MMAs (rows 0-127 and 128-255), which
//         cuts the shared-memory fill per FLOP by a third - the limit of the 128-row tile, whose operand
//         stream (48 KB per 4.2 MFLOP) cannot be kept in flight deep enough to cover the L2 latency.  The two
//         halves take all 512 tensor-memory columns, so the epilogue (eight warps) is not overlapped; the
//         producer still runs ahead into the next tile meanwhile.
// This removes the per-tile start-up bubbles of gemm_tc.cu's one-tile CTAs, which is what limits that kernel
// on compute-bound shapes.  Tiles are numbered with the M index fastest, so the CTAs that run side by side
// share one weight panel and the activation matrix stays in L2.
// Scope: tokens on the MMA M axis, tile-major 16-bit weights, no split-K, no fused all-reduce (those shapes
// stay with gemm_tc.cu).  Results and residuals that bulk copies can move go to the form with two CTAs to a tile
// (gemm_pair.cu, see gemm_ps_form): this one has the others and the grouped form.
//
// Grouped form (mixture of experts, rf_moe_grouped_gemm): the rows are (token, pick) pairs sorted by expert and
// the tile list comes from device memory - one entry {expert, first row, end row} per 128-row block of one
// expert's rows.  A tile reads its rows from the sorted activation matrix and its weight blocks from that
// expert's row tiles (up / gate projections) or k blocks (down projection) of the one packed expert bank; rows
// of the block that belong to the next expert are multiplied but never stored.  The number of tiles is only
// known on the device, so every CTA reads it there: the launch itself is shape-independent and graph-capturable.
#include "../common/dtype.cuh"
#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../rf_api.h"

namespace rf {

constexpr int kPsBM = 128, kPsBK = 64;
constexpr int kPsATile = kPsBM * kPsBK * 2;      // 16 KB
constexpr int kPsBlock = 128 * kPsBK * 2;        // one packed weight block
constexpr int kPsMaxStages = 8;
constexpr int kPsEpiBytes = 32 * 64 * 2;          // staging of one epilogue warp: 32 rows x 64 columns, 16-bit

struct GemmPsParams {
  void* out; int64_t ldo;
  const void* residual; int64_t ldr;
  const void* bias; const void* scale; const float* row_scale;
  const uint8_t* w_packed;
  int32_t* status;
  int M, N, k_blocks, bn, stages, act, dual_offset, dual_tiles;
  ActArgs act_args;
  int tiles_m, tiles_n;   // tiles_m counts tiles of 128*MT rows
  int band;               // row tiles per band of the tile order
  int pf_blocks;          // k blocks prefetched into L2 ahead of the ring
  int aff_vec;            // bias and scale may be read as 16-byte vectors (see finish16)
  int tma_out;            // results leave through shared-memory staging and tiled bulk stores
  // grouped form: grp[0] = number of row blocks, then {expert, row0, row_end, 0} per block (device memory)
  const int32_t* grp;
  int grp_rt_per_expert;  // row tiles of the weight image between two experts (projection whose N axis is split by expert)
  int grp_kb_per_expert;  // k blocks of the weight image between two experts (projection whose K axis is split by expert)
  int n_blocks;           // 128-row weight tiles of one matrix: a 256-wide column tile may end in the middle
  int kb_total;           // k blocks of a row tile of the whole weight image (stride between row tiles)
};

// Tile order: bands of `band` row tiles; inside a band the row index runs fastest and the weight panel
// advances slowly.  The CTAs that run side by side then share a few weight panels and one band of the
// activation matrix, and the band (sized to a fraction of L2) is reused from L2 by every panel of the sweep
// instead of being streamed from DRAM once per wave.
__device__ __forceinline__ void ps_tile_coords(const GemmPsParams& p, int tile, int* tm, int* tn) {
  const int per_band = p.band * p.tiles_n;
  const int b = tile / per_band, r = tile - b * per_band;
  const int rows_here = min(p.band, p.tiles_m - b * p.band);
  *tn = r / rows_here;
  *tm = b * p.band + r % rows_here;
}

// Coordinates of one tile: first activation row, end of the valid rows, weight column tile, and the offsets of
// the tile's expert inside the packed weight image (zero in the plain form).
struct PsTile { int row0, row_end, tm, tn, rt_add, kb_add; };
template <int MT>
__device__ __forceinline__ PsTile ps_tile(const GemmPsParams& p, int tile) {
  PsTile t;
  if (p.grp) {
    const int entry = tile / p.tiles_n;
    t.tn = tile - entry * p.tiles_n;
    const int e = p.grp[1 + 4 * entry];
    t.row0 = p.grp[2 + 4 * entry];
    t.row_end = p.grp[3 + 4 * entry];
    t.tm = 0;
    t.rt_add = e * p.grp_rt_per_expert;
    t.kb_add = e * p.grp_kb_per_expert;
  } else {
    ps_tile_coords(p, tile, &t.tm, &t.tn);
    t.row0 = t.tm * MT * kPsBM;
    t.row_end = p.M;
    t.rt_add = 0;
    t.kb_add = 0;
  }
  return t;
}

struct alignas(8) GemmPsCtl {
  uint64_t full[kPsMaxStages], empty[kPsMaxStages], acc_full[2], acc_empty[2], settled;
  uint32_t tmem_base;
  int32_t abort_flag, issued;                              // issued: k blocks that the producer has asked for
};

__device__ __forceinline__ uint4 shfl_u4(const uint4& q, int lane) {
  return make_uint4(__shfl_sync(0xffffffffu, q.x, lane), __shfl_sync(0xffffffffu, q.y, lane), __shfl_sync(0xffffffffu, q.z, lane),
                    __shfl_sync(0xffffffffu, q.w, lane));
}

// EXTRA: the epilogue has more to do than the activation (row scale, scale, bias, residual); without it their tests stay out of a
// loop whose length delays the MMA-issuing lane (3072 x 6144 x 1152, nothing to add: 40.5 -> 36.6 us)
template <typename T, bool DUAL, int MT, bool EXTRA>
__global__ void __launch_bounds__(64 + 128 * MT, 1)
gemm_ps_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmO, const GemmPsParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int bn = p.bn;
  constexpr int kW = DUAL ? 2 : 1;                         // weight tiles per stage
  const int b_bytes = bn * kPsBK * 2;
  constexpr int kAStage = MT * kPsATile;                   // activation bytes of one stage
  const int stage_bytes = kAStage + kW * b_bytes;
  const int half_cols = kW * bn;                           // TMEM columns of one 128-row half
  const int acc_cols = MT * half_cols;                     // ... of one accumulator buffer
  const int nbuf = 2 * acc_cols <= 512 ? 2 : 1;
  // after the ring: one 4 KB output staging buffer per epilogue warp, then the control block
  uint8_t* epi_stage = smem + (size_t)p.stages * stage_bytes;
  GemmPsCtl* ctl = reinterpret_cast<GemmPsCtl*>(epi_stage + 4 * MT * kPsEpiBytes);

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl->acc_full[b], 1);
      mbar_init(&ctl->acc_empty[b], 4 * MT);
    }
    mbar_init(&ctl->settled, 1);
    ctl->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    if (p.tma_out) tma_prefetch_desc(&tmO);
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, 512u);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  pdl_launch_dependents();         // after this CTA owns its TMEM columns
  volatile int32_t* abort_flag = &ctl->abort_flag;
  // Plain form: the tile count is a launch constant.  Grouped form: it (and the list) was written by the kernel
  // before this one, so it may only be read after the dependency wait; nothing of a tile is touched before that.
  auto tile_count = [&]() { return p.grp ? p.grp[0] * p.tiles_n : p.tiles_m * p.tiles_n; };

  // The producer's and the issuer's loops are run by their whole warp with one elected lane for the copies and MMAs (see gemm_tc.cu).
  uint64_t limit = kLocalWaitNs;
  if (warp == 0) {
    // ------------------------------------------------------------------ producer ----
    const bool lead = elect_one();
    const int nsub = bn / 128;
    auto load_w = [&](const PsTile& t, int kb, int s) {
      uint8_t* sb = smem + s * stage_bytes + kAStage;
#pragma unroll
      for (int wt = 0; wt < kW; ++wt)
        for (int sub = 0; sub < nsub; ++sub)             // behind the last weight tile: that tile once more, never stored
          bulk_load_1d(sb + wt * b_bytes + sub * kPsBlock,
                       p.w_packed + ((size_t)(min(t.tn * nsub + sub, p.n_blocks - 1) + t.rt_add + wt * p.dual_tiles) * p.kb_total + t.kb_add + kb) * kPsBlock,
                       kPsBlock, &ctl->full[s]);
    };
    auto load_x = [&](const PsTile& t, int kb, int s) {
#pragma unroll
      for (int h = 0; h < MT; ++h)   // a half wholly past the last row is zero-filled by the copy engine
        tma_load_2d(smem + s * stage_bytes + h * kPsATile, &tmA, &ctl->full[s], kb * kPsBK, t.row0 + h * kPsBM);
    };
    // L2 prefetch cursor: runs p.pf_blocks k blocks ahead of the ring (into the following tiles as well), so
    // the ring's own copies complete with L2 latency and the bytes in flight towards DRAM are not limited by
    // shared memory
    const int tiles = p.grp ? 0 : p.tiles_m * p.tiles_n;   // the prefetch cursor and the early ring fill are plain-form only
    int pf_tile = blockIdx.x, pf_kb = 0, pf_tm = 0, pf_tn = 0;
    if (pf_tile < tiles) ps_tile_coords(p, pf_tile, &pf_tm, &pf_tn);
    auto prefetch_next = [&](bool weights, bool acts) {
      if (pf_tile >= tiles) return;
      if (weights) {
        const int rt0 = pf_tn * nsub;
#pragma unroll
        for (int wt = 0; wt < kW; ++wt)
          for (int sub = 0; sub < nsub; ++sub)
            bulk_prefetch_l2(p.w_packed + ((size_t)(min(rt0 + sub, p.n_blocks - 1) + wt * p.dual_tiles) * p.k_blocks + pf_kb) * kPsBlock,
                             kPsBlock);
      }
      if (acts) {
#pragma unroll
        for (int h = 0; h < MT; ++h)
          if ((pf_tm * MT + h) * kPsBM < p.M) tma_prefetch_2d(&tmA, pf_kb * kPsBK, (pf_tm * MT + h) * kPsBM);
      }
      if (++pf_kb == p.k_blocks) {
        pf_kb = 0;
        pf_tile += gridDim.x;
        if (pf_tile < tiles) ps_tile_coords(p, pf_tile, &pf_tm, &pf_tn);
      }
    };
    // weights never depend on the previous kernel: the first ring fill starts before the dependency wait
    int tile = blockIdx.x;
    PsTile t = {};
    if (tile < tiles) t = ps_tile<MT>(p, tile);
    const int pre = tile < tiles ? min(p.stages, p.k_blocks) : 0;
    // the cursor passes the blocks the ring has just asked for, then takes its lead (weights only: the
    // activations may still be written by the previous kernel)
    const int ahead = p.pf_blocks > 0 ? pre + p.pf_blocks : 0;
    if (lead) {
      for (int i = 0; i < pre; ++i) {
        mbar_arrive_expect_tx(&ctl->full[i], (uint32_t)stage_bytes);
        load_w(t, i, i);
      }
      for (int i = 0; i < ahead; ++i) prefetch_next(i >= pre, false);
    }
    pdl_wait();
    if (lead)
      for (int i = 0; i < pre; ++i) load_x(t, i, i);
    const int ntiles = tile_count();
    const int total = tile < ntiles ? ((ntiles - 1 - tile) / (int)gridDim.x + 1) * p.k_blocks : 0;
    if (total && pre == 0) t = ps_tile<MT>(p, tile);
    int kb = pre, s = pre == p.stages ? 0 : pre;
    uint32_t phase = pre == p.stages ? 0 : 1;              // a stage's first release completes phase 0; before it nothing is waited for
    int i = pre;
    for (; i < total; ++i, ++kb) {
      if (kb == p.k_blocks) {
        kb = 0;
        tile += gridDim.x;
        t = ps_tile<MT>(p, tile);
      }
      const bool free = role_wait(&ctl->empty[s], phase, &limit, &ctl->abort_flag, p.status, kStatusTmaTimeout, kTagGemmTc, i);
      if (free && lead) {
        mbar_arrive_expect_tx(&ctl->full[s], (uint32_t)stage_bytes);
        load_w(t, kb, s);
        load_x(t, kb, s);
        if (p.pf_blocks > 0) prefetch_next(true, true);
      }
      if (!agreed(free)) break;
      if (++s == p.stages) { s = 0; phase ^= 1u; }
    }
    if (lead) ctl->issued = i;
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer ----
    pdl_wait();
    const bool lead = elect_one();
    const uint32_t idesc = umma_idesc_f16(kPsBM, bn, Num<T>::kFmt);
    // operand descriptors advance by constants (16-byte units)
    const uint64_t a_desc = umma_desc_k128(smem_u32(smem)), b_desc = umma_desc_k128(smem_u32(smem) + kAStage);
    const uint32_t stage_step = (uint32_t)(stage_bytes >> 4), b_second = (uint32_t)(b_bytes >> 4);
    int s = 0, lt = 0;
    uint32_t phase = 0, at = 0;
    const int tiles = tile_count();
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++lt) {
      const int b = nbuf == 2 ? lt & 1 : 0;
      if (!agreed(role_wait(&ctl->acc_empty[b], ((uint32_t)(nbuf == 2 ? lt >> 1 : lt) & 1u) ^ 1u, &limit, &ctl->abort_flag, p.status, kStatusMmaTimeout, kTagGemmTc, lt) && limit)) break;
      tc_fence_after_sync();
      const uint32_t acc = tmem_base + (uint32_t)(b * acc_cols);
      for (int kb = 0; kb < p.k_blocks; ++kb) {
        role_wait(&ctl->full[s], phase, &limit, &ctl->abort_flag, p.status, kStatusMmaTimeout, kTagGemmTc, lt);
        tc_fence_after_sync();
        if (lead) {
          const uint64_t da = a_desc + at, db = b_desc + at;
#pragma unroll
          for (int k = 0; k < kPsBK / 16; ++k) {
            const uint32_t accum = k > 0 ? 1u : (kb > 0 ? 1u : 0u);
#pragma unroll
            for (int h = 0; h < MT; ++h) {
              umma_f16(acc + h * half_cols, da + (h * (kPsATile >> 4) + 2 * k), db + 2 * k, idesc, accum);
              if (DUAL) umma_f16(acc + h * half_cols + bn, da + (h * (kPsATile >> 4) + 2 * k), db + (b_second + 2 * k), idesc, accum);
            }
          }
          if (limit) umma_commit(&ctl->empty[s]);
        }
        at += stage_step;
        if (++s == p.stages) { s = 0; at = 0; phase ^= 1u; }
      }
      if (lead) umma_commit(&ctl->acc_full[b]);
    }
  } else {
    // ------------------------------------------------------------------ epilogue ----
    pdl_wait();
    const int quarter = warp & 3;                          // the TMEM lanes a warp may read
    const int half = (warp - 2) >> 2;                      // which 128-row half of the tile it drains
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const T* bias = EXTRA ? reinterpret_cast<const T*>(p.bias) : nullptr;
    const T* scale = EXTRA ? reinterpret_cast<const T*>(p.scale) : nullptr;
    const T* resid = EXTRA ? reinterpret_cast<const T*>(p.residual) : nullptr;
    T* out = reinterpret_cast<T*>(p.out);
    const int N = p.N;
    const bool out_vec = (p.ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const bool res_vec = (p.ldr & 7) == 0 && (reinterpret_cast<uintptr_t>(resid) & 15) == 0;
    int lt = 0;
    const int tiles = tile_count();
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++lt) {
      const int b = lt % nbuf;
      const PsTile pt = ps_tile<MT>(p, tile);
      const int tn = pt.tn;
      const int M = pt.row_end;                            // rows at and past it are not this tile's to store
      const int row = pt.row0 + half * kPsBM + r;
      const int n_base = tn * bn;
      // Bias and scale of the tile's columns, eight to a lane, and the row's first residual values are asked for before the accumulator
      // is awaited: next to the operand ring there is no L1 to speak of, and a load inside the column loop is a trip to L2
      // (3072 x 6144 x 1152 with a bias, us: sixteen two-byte loads per 16 columns 69.8, two 16-byte ones 48.0, this 42.3, no bias 35.9).
      uint4 bias_g = {}, bias_u = {}, scale_g = {}, scale_u = {}, rv[DUAL ? 2 : 1][2] = {};
      if constexpr (EXTRA) {
        const int n = n_base + lane * 8;
        if (lane * 8 < bn) {
          if (bias) bias_g = vec8_upto(bias, n, N, p.aff_vec);
          if (scale) scale_g = vec8_upto(scale, n, N, p.aff_vec);
          if (DUAL && bias) bias_u = vec8_upto(bias + p.dual_offset, n, N, p.aff_vec);
          if (DUAL && scale) scale_u = vec8_upto(scale + p.dual_offset, n, N, p.aff_vec);
        }
        if (resid && row < M) {
#pragma unroll
          for (int q = 0; q < (DUAL ? 4 : 2); ++q) rv[q >> 1][q & 1] = vec8_upto(resid + (size_t)row * p.ldr, n_base + q * 8, N, res_vec);
        }
      }
      const bool have = role_wait(&ctl->acc_full[b], (uint32_t)(lt / nbuf) & 1u, &limit, &ctl->abort_flag, p.status, kStatusEpilogueTimeout, kTagGemmTc, tile);
      if (!agreed(have && !*abort_flag)) break;
      tc_fence_after_sync();
      const uint32_t acc = lane_base + (uint32_t)(b * acc_cols + half * half_cols);
      const float rs = (EXTRA && p.row_scale && row < M) ? p.row_scale[row] : 1.f;
      // Output path: 64 finished columns of the warp's 32 rows are parked in a swizzled staging tile and leave as ONE tiled bulk
      // store issued by lane 0 - whole 128-byte lines, asynchronous, no store instructions on the epilogue warps (16-byte stores
      // to 32 rows per instruction kept the store queue saturated: 537 MB on the L1->L2 path for 67 MB of output).
      uint8_t* stg = epi_stage + (size_t)(warp - 2) * kPsEpiBytes;
      const int row0 = pt.row0 + half * kPsBM + quarter * 32;
      // grouped form: rows behind the expert's last one are another expert's, so only whole 32-row pieces leave this way
      const bool tma_out = p.tma_out != 0 && (!p.grp || row0 + 32 <= M);
      auto chunk_begin = [&]() {                       // the previous bulk store has read the staging tile
        if (lane == 0) bulk_wait_read_all();
        __syncwarp();
      };
      auto chunk_end = [&](int c_first) {              // c_first: first column of the 64-column chunk in the tile
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && row0 < M && n_base + c_first < N) {
          tma_store_2d(&tmO, stg, n_base + c_first, row0);
          bulk_commit_group();
        }
      };
      // 16 residual values of this row (zeros where there are none): added in fp32 and rounded once
      auto resid16 = [&](int n0, uint4 (&rv)[2]) {
        rv[0] = rv[1] = make_uint4(0u, 0u, 0u, 0u);
        if (!resid || row >= M) return;
        rv[0] = vec8_upto(resid + (size_t)row * p.ldr, n0, N, res_vec);
        rv[1] = vec8_upto(resid + (size_t)row * p.ldr, n0 + 8, N, res_vec);
      };
      // x <- x * scale + bias for 16 columns; every lane must take part (the tile's values lie eight to a lane)
      auto affine16 = [&](int c0, float (&x)[16], const uint4& sq, const uint4& bq) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int src = (c0 >> 3) + h;
          float f[8];
          if (scale) {
            const uint4 q = shfl_u4(sq, src);
            unpack8<T>(q, f);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[h * 8 + j] *= f[j];
          }
          if (bias) {
            const uint4 q = shfl_u4(bq, src);
            unpack8<T>(q, f);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[h * 8 + j] += f[j];
          }
        }
      };
      auto finish16 = [&](int c0, const uint32_t* g16, const uint32_t* u16, const uint4 (&rv)[2]) {
        const int n0 = n_base + c0;
        float g[16], u[16], v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          g[j] = __uint_as_float(g16[j]);
          u[j] = DUAL ? __uint_as_float(u16[j]) : 0.f;
        }
        if constexpr (EXTRA) {
          if (p.row_scale) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              g[j] *= rs;
              if (DUAL) u[j] *= rs;
            }
          }
          affine16(c0, g, scale_g, bias_g);
          if (DUAL) affine16(c0, u, scale_u, bias_u);
        }
        if (!tma_out && (row >= M || n0 >= N)) return;
        apply_act_n<16>(p.act, g, u, v, p.act_args);
        float lo[8], hi[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) { lo[j] = v[j]; hi[j] = v[8 + j]; }
        if constexpr (EXTRA) {
          if (resid) {
            float r0[8], r1[8];
            unpack8<T>(rv[0], r0);
            unpack8<T>(rv[1], r1);
#pragma unroll
            for (int j = 0; j < 8; ++j) { lo[j] += r0[j]; hi[j] += r1[j]; }
          }
        }
        if (tma_out) {
          // row `lane` of the warp's staging tile, 128-byte swizzled as the bulk store expects it
          const int ch = (c0 >> 3) & 7;
          store8(reinterpret_cast<T*>(stg + lane * 128 + ((ch ^ (lane & 7)) << 4)), lo);
          store8(reinterpret_cast<T*>(stg + lane * 128 + (((ch + 1) ^ (lane & 7)) << 4)), hi);
        } else if (out_vec && n0 + 16 <= N) {
          store8(out + (size_t)row * p.ldo + n0, lo);
          store8(out + (size_t)row * p.ldo + n0 + 8, hi);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (n0 + j < N) out[(size_t)row * p.ldo + n0 + j] = Num<T>::from_f(j < 8 ? lo[j & 7] : hi[j & 7]);
        }
      };
      // 16 columns (of each accumulator) per tensor-memory round trip for one accumulator and 32 for the GLU pair.  Measured
      // alternatives: 32- and 64-column trips 1 - 5 % slower, a shared-memory transpose for full-line stores 35 % slower - long
      // instruction bursts of the epilogue warps delay the single MMA-issuing lane that shares their schedulers.
      constexpr int kTrip = DUAL ? 32 : 16;
      for (int c0 = 0; c0 < bn; c0 += kTrip) {
        uint32_t ra[kTrip], rb[kTrip];
        uint4 rnext[kTrip / 16][2];
        if constexpr (DUAL) {
          tmem_ld32(acc + c0, *reinterpret_cast<uint32_t(*)[32]>(&ra[0]));
          tmem_ld32(acc + bn + c0, *reinterpret_cast<uint32_t(*)[32]>(&rb[0]));
        } else {
          tmem_ld16(acc + c0, *reinterpret_cast<uint32_t(*)[16]>(&ra[0]));
        }
        if constexpr (EXTRA) {                         // the next trip's residual values
#pragma unroll
          for (int q = 0; q < kTrip / 16; ++q) resid16(c0 + kTrip < bn ? n_base + c0 + kTrip + q * 16 : N, rnext[q]);
        }
        tmem_ld_wait();
        if (tma_out && (c0 & 63) == 0) chunk_begin();
#pragma unroll
        for (int q = 0; q < kTrip / 16; ++q) finish16(c0 + q * 16, ra + q * 16, DUAL ? rb + q * 16 : ra, rv[q]);
        if (tma_out && ((c0 + kTrip) & 63) == 0) chunk_end(c0 + kTrip - 64);
        if constexpr (EXTRA) {
#pragma unroll
          for (int q = 0; q < kTrip / 16; ++q) { rv[q][0] = rnext[q][0]; rv[q][1] = rnext[q][1]; }
        }
      }
      // this accumulator buffer may now be overwritten by a later tile
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->acc_empty[b]);
    }
    if (p.tma_out && lane == 0) bulk_wait_all();       // the last stores are complete before the CTA retires
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {                                       // a role gave up: what the others had started ends first
    if (warp == 0) settle_copies(ctl->full, p.stages, ctl->issued);
    if (warp == 1) settle_mmas(&ctl->settled);
  }
  if (warp == 1) tmem_dealloc(tmem_base, 512u);
}

int ps_forced_band() {
  static const int band = [] { const char* e = getenv("RF_GEMM_PS_BAND"); return e ? atoi(e) : 0; }();
  return band;
}

template <typename T, bool DUAL, int MT, bool EXTRA>
static int launch_ps(const RfGemm* g, int bn, cudaStream_t stream) {
  auto kfn = gemm_ps_kernel<T, DUAL, MT, EXTRA>;
  RF_ALLOW_SMEM_PER_DEVICE(kfn, 227 * 1024);
  CUtensorMap tmA, tmO;
  int rc = make_tmap_2d(&tmA, g->x, g->dtype, 2, g->K, g->M, g->ldx, kPsBK, kPsBM, true);
  if (rc) return rc;
  static const bool tma_out_enabled = [] { const char* e = getenv("RF_GEMM_PS_TMA_OUT"); return !(e && e[0] == '0'); }();
  const bool tma_out = tma_out_enabled && (g->ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(g->out) & 15) == 0;
  if (tma_out) {
    rc = make_tmap_2d(&tmO, g->out, g->dtype, 2, g->N, g->M, g->ldo, 64, 32, true);
    if (rc) return rc;
  } else {
    tmO = tmA;
  }
  GemmPsParams p = {};
  p.out = g->out; p.ldo = g->ldo; p.residual = g->residual; p.ldr = g->ldr;
  p.bias = g->bias; p.scale = g->scale; p.row_scale = g->row_scale;
  p.w_packed = reinterpret_cast<const uint8_t*>(g->w);
  p.status = g->status;
  p.aff_vec = ((reinterpret_cast<uintptr_t>(g->bias) | reinterpret_cast<uintptr_t>(g->scale)) & 15) == 0 && (g->dual_offset & 7) == 0;
  p.tma_out = tma_out ? 1 : 0;
  p.M = g->M; p.N = g->N; p.k_blocks = ceil_div(g->K, kPsBK); p.bn = bn;
  p.kb_total = p.k_blocks; p.n_blocks = ceil_div(g->N, 128);
  p.act = g->act; p.act_args = {g->act_limit, g->act_alpha}; p.dual_offset = g->dual_offset; p.dual_tiles = ceil_div(g->N, 128);
  p.tiles_m = ceil_div(g->M, kPsBM * MT); p.tiles_n = ceil_div(g->N, bn);
  const int stage_bytes = MT * kPsATile + (DUAL ? 2 : 1) * bn * kPsBK * 2;
  {
    // a band of activation rows of about 16 MB: it and a weight matrix of a few tens of MB stay in L2 together
    const int64_t row_tile_bytes = (int64_t)kPsBM * MT * g->K * 2;
    p.band = (int)std::max<int64_t>(1, std::min<int64_t>(p.tiles_m, (16ll << 20) / std::max<int64_t>(1, row_tile_bytes)));
    if (ps_forced_band() > 0) p.band = std::min(p.tiles_m, ps_forced_band());
    static const int pf_kb = [] { const char* e = getenv("RF_GEMM_L2_PREFETCH_KB"); return e ? atoi(e) : 0; }();
    p.pf_blocks = std::min(16, pf_kb * 1024 / stage_bytes);
  }
  const int ctl_bytes = (int)sizeof(GemmPsCtl) + 1024 /*alignment slack*/ + 4 * MT * kPsEpiBytes;
  p.stages = std::min(kPsMaxStages, (227 * 1024 - ctl_bytes) / stage_bytes);
  RF_REQUIRE(p.stages >= 2, "persistent GEMM: a %d-byte stage does not fit twice in shared memory", stage_bytes);
  const size_t smem = (size_t)p.stages * stage_bytes + ctl_bytes;
  const int grid = std::min(p.tiles_m * p.tiles_n, sm_count());
  RF_CUDA_CHECK(::rf::launch_k(kfn, dim3(grid), dim3(64 + 128 * MT), smem, stream, 1, tmA, tmO, p));
  ::rf::count_launch();
  return RF_OK;
}

// Tile shape of a launch and its estimated time.
struct PsShape { int bn, rows; long ns; };

// The main loop of a tile is bound by its operand stream, not by the tensor core: per 64-column k block and SM, with all SMs busy,
// 128 x 128 tiles take 450 ns (32 KB), 256 x 128 and 128 x 256 tiles 595 ns (48 KB, twice the work), 256 x 256 tiles 800 ns
// (64 KB, four times the work).  So larger tiles win unless they leave SMs without one: a launch takes as many waves of them as
// the busiest SM has tiles.  Tiles that take all of tensor memory (512 columns) also wait for their epilogue, about 3.5 us, each;
// the others only for the last one.  fp16, us, 128-row / 256-row tiles 128 wide (model in brackets): 3072 x 1152 x 4304 60.4 / 39.9
// (65 / 44), 768 x 4304 x 1152 19.7 / 15.0 (21 / 15); 3072 x 6144 x 1152 with 256 x 256 tiles 37.3 (39).
static int ps_forced_rows() {
  static const int rows = [] { const char* e = getenv("RF_GEMM_PS_ROWS"); return e ? atoi(e) : 0; }();
  return rows;
}
static PsShape ps_shape(const RfGemm* g) {
  const bool dual = g->dual_offset > 0;
  const int k_blocks = ceil_div(g->K, kPsBK), sms = sm_count(), forced = ps_forced_rows();
  PsShape best = {0, 0, 0};
  for (int mt = 2; mt >= 1; --mt) {
    if ((forced == 128 || forced == 256) && forced != mt * kPsBM) continue;
    for (int bn = dual || g->N <= 128 ? 128 : 256; bn >= 128; bn -= 128) {   // a 256-wide tile may end in the middle
      const long tiles = (long)ceil_div(g->M, mt * kPsBM) * ceil_div(g->N, bn), waves = (tiles + sms - 1) / sms;
      const int pieces = mt + (dual ? 2 : bn / 128);                         // 16 KB operand pieces of a stage
      const long kb_ns = pieces == 2 ? 450 : pieces == 3 ? 595 : 800;
      const bool alone = mt * bn * (dual ? 2 : 1) > 256;
      const long ns = 3000 + waves * k_blocks * kb_ns + (alone ? waves * 3500 : (dual ? 256 : bn) * 9);
      if (best.bn == 0 || ns < best.ns) best = {bn, mt * kPsBM, ns};
    }
  }
  // 256 x 128 and 128 x 256 tiles move the same pieces, but a stage of the latter has one row piece to wait for and its MMAs are twice as wide: 9 %
  // off a k block.  Its four epilogue warps have twice the columns each, which shows behind short rows, longer ones if there is more to do than the
  // activation (fp16, us, 256 x 128 / 128 x 256: 825 x 4096 x 12288 101 / 91, 3072 x 1152 x 4304 39.0 / 35.9, 1300 x 2048 x 2048 21.4 / 20.3; bf16
  // 6600 x 2048 x 1024 30.3 / 28.4, x 512 18.4 / 18.9, x 128 10.9 / 15.2; with bias and residual 825 x 4096 x 12288 105 / 95, 825 x 4096 x 4096
  // 40.9 / 38.5, 1300 x 2560 x 2560 28.7 / 28.5, 1300 x 2048 x 2048 24.2 / 25.0).
  const bool extra = g->bias || g->scale || g->row_scale || g->residual;
  auto rounds = [&](int rows, int cols) { return ceil_div(ceil_div(g->M, rows) * ceil_div(g->N, cols), sms); };
  if (forced == 0 && !dual && best.rows == 256 && best.bn == 128 && g->N > 128 && k_blocks >= (extra ? 48 : 16) && rounds(128, 256) <= rounds(256, 128))
    best = {256, 128, best.ns};
  return best;
}

long gemm_pair_ns(const RfGemm* g);                              // gemm_pair.cu: the form with two CTAs to a tile
int launch_gemm_pair(const RfGemm* g, cudaStream_t stream);

// Whether the form with two CTAs to a tile may be chosen: not where the environment turns the persistent kernels off or sets the rows of a tile.
bool gemm_pairs_on() {
  static const bool on = [] { const char* e = getenv("RF_GEMM_PERSISTENT"); return !(e && e[0] == '0'); }();
  return on && ps_forced_rows() != 128 && ps_forced_rows() != 256;
}

// Which persistent kernel takes this GEMM (called by rf_gemm after its argument checks, with the tile kernel's plan): 0 neither, 1 the one with a
// CTA to a tile, 2 CTA pairs, wherever their bulk copies can write the result and read the residual (fp16, us, one CTA / two to a tile:
// 3072 x 4304 x 1152 32.3 / 25, 4770 x 2048 x 2048 50.8 / 33.2, 825 x 2048 x 8192 50.8 / 28.6, 4770 x 16384 x 2048 SwiGLU 626 / 416).
// Weights on the rows (at most 256 tokens): 129 to 256 tokens of short K, where one row tile of the CTA pairs does without the tile kernel's reduction over
// splits.  fp16, us, tile / pairs: 200 x 2048 x 2048 13.7 / 9.3, 200 x 8192 x 2048 GLU 34.3 / 21.8; 200 x 4096 x 4096 18.3 / 20.8, 200 x 1152 x 4304
// 16.2 / 16.6, 200 x 2048 x 8192 21.3 / 28.1.
// Tokens on the rows: where it is estimated to be no slower than
// the one-tile kernel with `splits` K splits, whose CTAs pay the same per k block (two of them share an SM's operand stream), about
// 4.5 us around it and 6.5 us more for the reduction of a split (fp16, us, persistent / split kernel: 825 x 2560 x 2048 20 / 26,
// 825 x 2048 x 2048 20 / 30; 768 x 1152 x 4304 34 / 23, 825 x 2048 x 16384 119 / 96).
int gemm_ps_form(const RfGemm* g, bool swap, int splits, int bn, int tiles) {
  static const bool enabled = [] { const char* e = getenv("RF_GEMM_PERSISTENT"); return !(e && e[0] == '0'); }();
  if (!enabled || g->ar_world > 1 || !g->w_packed || g->w_int8 || g->force_splits || g->force_bn) return 0;
  const long pairs_ns = gemm_pair_ns(g);
  if (swap) return g->M > 128 && g->M <= 256 && g->K <= 2048 && g->force_swap < 0 && pairs_ns ? 2 : 0;
  // Up to 255 columns that the tile kernel can split along K are left to it by the other form's estimate: few pairs have a tile.  That rests on
  // one size, 4770 x 128 x 2048, tile / pairs 17 / 18 us, and on results staying what they were for routers of few experts.
  const long pair_ns = splits > 1 && g->N < 256 ? 0 : pairs_ns;
  const PsShape s = ps_shape(g);
  if (s.bn == 0) return 0;
  const long sms = sm_count(), ctas = (long)tiles * splits, kb = ceil_div(ceil_div(g->K, kPsBK), splits);
  const long kb_ns = (g->dual_offset > 0 || bn > 128) ? 595 : 450;
  const long load = splits == 1 ? (ctas + sms - 1) / sms * 100 : std::max(100l, ctas * 100 / sms);    // busiest SM's CTAs, per cent
  if ((pair_ns ? std::min(pair_ns, s.ns) : s.ns) > 4500 + (splits > 1 ? 6500 : 0) + kb * kb_ns * load / 100) return 0;
  return pairs_ns ? 2 : 1;
}

template <typename T, bool EXTRA>
static int launch_ps_t(const RfGemm* g, bool dual, int bn, int rows, cudaStream_t stream) {
  if (rows == 256) return dual ? launch_ps<T, true, 2, EXTRA>(g, bn, stream) : launch_ps<T, false, 2, EXTRA>(g, bn, stream);
  return dual ? launch_ps<T, true, 1, EXTRA>(g, bn, stream) : launch_ps<T, false, 1, EXTRA>(g, bn, stream);
}

// `form`: what gemm_ps_form said.
int launch_gemm_ps(const RfGemm* g, int form, cudaStream_t stream) {
  if (form == 2) return launch_gemm_pair(g, stream);
  const bool dual = g->dual_offset > 0;
  const PsShape s = ps_shape(g);
  const bool extra = g->bias || g->scale || g->row_scale || g->residual;
  if (g->dtype == 0)
    return extra ? launch_ps_t<__half, true>(g, dual, s.bn, s.rows, stream) : launch_ps_t<__half, false>(g, dual, s.bn, s.rows, stream);
  return extra ? launch_ps_t<__nv_bfloat16, true>(g, dual, s.bn, s.rows, stream) : launch_ps_t<__nv_bfloat16, false>(g, dual, s.bn, s.rows, stream);
}

// Grouped (mixture-of-experts) launch: see the file comment.  One accumulator or a GLU pair, 128-row tiles.
template <typename T, bool DUAL, bool EXTRA>
static int launch_ps_grouped(const RfMoeGroupedGemm* a, cudaStream_t stream) {
  auto kfn = gemm_ps_kernel<T, DUAL, 1, EXTRA>;
  RF_ALLOW_SMEM_PER_DEVICE(kfn, 227 * 1024);
  CUtensorMap tmA, tmO;
  int rc = make_tmap_2d(&tmA, a->x, a->dtype, 2, a->K, a->max_rows, a->ldx, kPsBK, kPsBM, true);
  if (rc) return rc;
  const bool tma_out = (a->ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(a->out) & 15) == 0;
  if (tma_out) {
    rc = make_tmap_2d(&tmO, a->out, a->dtype, 2, a->N, a->max_rows, a->ldo, 64, 32, true);
    if (rc) return rc;
  } else {
    tmO = tmA;
  }
  const int bn = !DUAL && (a->N % 256 == 0 || a->N >= 1024) ? 256 : 128;
  GemmPsParams p = {};
  p.out = a->out; p.ldo = a->ldo;
  p.row_scale = a->row_scale;
  p.w_packed = reinterpret_cast<const uint8_t*>(a->w);
  p.status = a->status;
  p.M = a->max_rows; p.N = a->N; p.k_blocks = ceil_div(a->K, kPsBK); p.bn = bn;
  p.act = a->act; p.act_args = {a->act_limit, a->act_alpha}; p.dual_offset = DUAL ? a->N : 0; p.dual_tiles = a->bank_section_row_tiles;
  p.tiles_m = 0; p.tiles_n = ceil_div(a->N, bn);
  p.band = 1;
  p.tma_out = tma_out ? 1 : 0;
  p.grp = a->tiles; p.grp_rt_per_expert = a->rt_per_expert; p.grp_kb_per_expert = a->kb_per_expert;
  p.kb_total = a->bank_kb_total; p.n_blocks = ceil_div(a->N, 128);
  const int stage_bytes = kPsATile + (DUAL ? 2 : 1) * bn * kPsBK * 2;
  const int ctl_bytes = (int)sizeof(GemmPsCtl) + 1024 + 4 * kPsEpiBytes;
  p.stages = std::min(kPsMaxStages, (227 * 1024 - ctl_bytes) / stage_bytes);
  const size_t smem = (size_t)p.stages * stage_bytes + ctl_bytes;
  RF_CUDA_CHECK(::rf::launch_k(kfn, dim3(sm_count()), dim3(64 + 128), smem, stream, 1, tmA, tmO, p));
  ::rf::count_launch();
  return RF_OK;
}

template <typename T>
static int launch_ps_grouped_t(const RfMoeGroupedGemm* a, cudaStream_t stream) {
  if (a->row_scale) return a->dual ? launch_ps_grouped<T, true, true>(a, stream) : launch_ps_grouped<T, false, true>(a, stream);
  return a->dual ? launch_ps_grouped<T, true, false>(a, stream) : launch_ps_grouped<T, false, false>(a, stream);
}

int launch_moe_grouped(const RfMoeGroupedGemm* a, cudaStream_t stream) {
  return a->dtype == 0 ? launch_ps_grouped_t<__half>(a, stream) : launch_ps_grouped_t<__nv_bfloat16>(a, stream);
}

// int8 tile-major weight image -> 16-bit tile-major image (the 128-byte-swizzled block layout the MMA reads).
// One thread widens eight values: 8 bytes in, 16 bytes out.  Exact in fp16 and bf16 (|q| <= 127).
template <typename T>
__global__ void widen_packed_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t pieces) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pieces; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t block = i >> 10;                     // 128 rows x 8 pieces
    const int row = (int)(i & 1023) >> 3, c = (int)(i & 7);
    const uint2 q = *reinterpret_cast<const uint2*>(src + block * 8192 + row * 64 + c * 8);
    *reinterpret_cast<uint4*>(dst + block * 16384 + row * 128 + ((c ^ (row & 7)) << 4)) = widen_i8x8<T>(q);
  }
}

int widen_packed(const void* src, void* dst, int64_t blocks, int dtype, cudaStream_t stream) {
  const int64_t pieces = blocks * 1024;
  const int grid = (int)std::min<int64_t>((pieces + 255) / 256, (int64_t)sm_count() * 16);
  // no programmatic dependent launch here: the GEMM that follows prefetches this image before its dependency wait
  const uint8_t* sp = reinterpret_cast<const uint8_t*>(src);
  uint8_t* dp = reinterpret_cast<uint8_t*>(dst);
  if (dtype == 0) RF_CUDA_CHECK(::rf::launch_serial(widen_packed_kernel<__half>, dim3(grid), dim3(256), 0, stream, sp, dp, pieces));
  else RF_CUDA_CHECK(::rf::launch_serial(widen_packed_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, stream, sp, dp, pieces));
  ::rf::count_launch();
  return RF_OK;
}

}  // namespace rf

extern "C" int rf_moe_grouped_gemm(const RfMoeGroupedGemm* a, rf_stream_t stream) {
  RF_SKIP_IF_REPLAYING();
  RF_REQUIRE(a && a->x && a->w && a->out && a->tiles, "moe_grouped_gemm needs x, w, out and the tile list");
  RF_REQUIRE(a->max_rows > 0 && a->N > 0 && a->K > 0 && a->K % 8 == 0 && a->ldx % 8 == 0, "moe_grouped_gemm shape %d x %d x %d",
             a->max_rows, a->N, a->K);
  RF_REQUIRE(a->dtype == 0 || a->dtype == 1, "moe_grouped_gemm dtype");
  RF_REQUIRE(a->bank_kb_total > 0 && a->rt_per_expert >= 0 && a->kb_per_expert >= 0, "moe_grouped_gemm bank geometry");
  RF_REQUIRE((reinterpret_cast<uintptr_t>(a->w) & 127) == 0, "packed expert bank must be 128-byte aligned");
  if (a->dual) RF_REQUIRE(a->bank_section_row_tiles > 0 && rf::act_is_dual(a->act), "a GLU grouped GEMM needs the section size and an activation of two operands");
  if (a->act == rf::kActClippedGlu) RF_REQUIRE(a->act_limit > 0.f, "this activation needs a positive limit");
  return rf::launch_moe_grouped(a, static_cast<cudaStream_t>(stream));
}
