// Persistent tcgen05 GEMM on CTA pairs:  out[M,N] = epilogue( x[M,K] . w[N,K]^T ), tokens on the MMA rows, tile-major 16-bit weights.
//
// Two CTAs of a cluster (the two SMs of a TPC) share one 256 x BN tile: each loads 128 activation rows and HALF of the tile's weight
// rows, the even CTA issues one 256-row MMA per 16 columns of K for both (cta_group::2), and each drains the 128 x BN accumulator of its own
// rows.  A GLU pair is the same with BN = 256: the even CTA brings the gate's 128 weight rows, the odd one those of the up projection.
// Against one CTA per tile (gemm_ps.cu) this
//   * moves 32 KB per 64-column k block for 128 x 256 results of an SM instead of 48 KB;
//   * leaves room for two accumulators of 256 columns, so the epilogue always runs under the next tile's MMAs;
//   * has half as many barriers and commits per result, and those bound a k block that the tensor core is through with in 270 ns.
// Roles per CTA: warp 0 loads (five or six stages), warp 1 of the even CTA issues MMAs, eight warps drain: two for each 32 rows, 64
// columns at a time.  A chunk's residual arrives by a bulk tensor load in the staging tile that the result then leaves from.
#include <algorithm>

#include "../common/dtype.cuh"
#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../rf_api.h"

namespace rf {

constexpr int kPrBM = 128, kPrBK = 64;           // activation rows of one CTA, columns of a k block
constexpr int kPrPiece = 128 * kPrBK * 2;        // 16 KB: 128 rows of a k block
constexpr int kPrMaxStages = 8, kPrEpiWarps = 8;
constexpr int kPrChunk = 32 * 64 * 2;            // 32 rows x 64 columns of 16-bit results

struct GemmPairParams {
  const void* bias; const void* scale; const float* row_scale;
  int32_t* status;
  int M, N, k_blocks, bn, stages, act, dual_offset;
  ActArgs act_args;
  int tiles_m, tiles_n, band;
  int n_blocks;           // 128-row blocks of one weight matrix
  int residual;           // tmR is the residual's map
};

struct alignas(8) GemmPairCtl {
  uint64_t full[kPrMaxStages], empty[kPrMaxStages], acc_full[2], acc_empty[2], res[kPrEpiWarps][2], settled;
  uint32_t tmem_base;
  int32_t gave_up;                                         // a role of either CTA did (see role_wait)
};

// Bands of row tiles, row index fastest inside a band (see gemm_ps.cu): the pairs that run side by side share a few weight panels.
__device__ __forceinline__ void pair_tile_coords(const GemmPairParams& p, int tile, int* tm, int* tn) {
  const int per_band = p.band * p.tiles_n;
  const int b = tile / per_band, r = tile - b * per_band;
  const int rows_here = min(p.band, p.tiles_m - b * p.band);
  *tn = r / rows_here;
  *tm = b * p.band + r % rows_here;
}

// A role of one CTA gave up and all of both have stopped: what they had started ends first.  A copy completes on the even CTA's barrier, in a phase
// that lacks an arrival where only one of the two had asked for its stage, so copies (residuals among them) get their time by the clock.
static __device__ __noinline__ void settle_pair(uint64_t* settled, uint32_t rank, int warp) {
  if (warp == 0) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < kSettleNs) __nanosleep(1000);
  } else if (warp == 1 && rank == 0) {
    if (elect_one()) pair_umma_commit(settled, 1);
    __syncwarp();
    mbar_wait(settled, 0, kSettleNs);
  }
  __syncwarp();
  cluster_sync_all();
}

// EXTRA: scale, bias or row scale (the residual is handled either way)
template <typename T, bool DUAL, bool EXTRA>
__global__ void __launch_bounds__(64 + 32 * kPrEpiWarps, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW32,
                 const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmR, const GemmPairParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const int acc_cols = DUAL ? 256 : p.bn;                  // columns of an accumulator
  const int w_rows = acc_cols / 2;                         // weight rows of this CTA
  const int stage_bytes = kPrPiece + w_rows * kPrBK * 2;
  uint8_t* epi_stage = smem + (size_t)p.stages * stage_bytes;
  GemmPairCtl* ctl = reinterpret_cast<GemmPairCtl*>(epi_stage + kPrEpiWarps * 2 * kPrChunk);

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl->acc_full[b], 1);
      mbar_init(&ctl->acc_empty[b], 2 * kPrEpiWarps);
      for (int w = 0; w < kPrEpiWarps; ++w) mbar_init(&ctl->res[w][b], 1);
    }
    mbar_init(&ctl->settled, 1);
    ctl->gave_up = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmO);
  }
  __syncwarp();
  if (warp == 1) {
    pair_tmem_alloc(&ctl->tmem_base, 512u);
    pair_tmem_relinquish();
  }
  tc_fence_before_sync();
  cluster_sync_all();                                      // both CTAs' barriers stand and both own their tensor memory
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  pdl_launch_dependents();
  const int tiles = p.tiles_m * p.tiles_n, first = blockIdx.x >> 1, step = gridDim.x >> 1;
  uint64_t limit = kLocalWaitNs;
  volatile int32_t* gave_up = &ctl->gave_up;
  const uint32_t peer_gave_up = dsmem_addr(smem_u32(&ctl->gave_up), rank ^ 1u);
  auto wait = [&](uint64_t* bar, uint32_t parity, int32_t code, int32_t detail) {
    return role_wait(bar, parity, &limit, &ctl->gave_up, p.status, code, kTagGemmTc, detail, 0, peer_gave_up);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer ----
    const bool lead = elect_one();
    const int total = first < tiles ? ((tiles - 1 - first) / step + 1) * p.k_blocks : 0;     // k blocks of this pair
    const uint32_t full0 = dsmem_addr(smem_u32(&ctl->full[0]), 0);                           // the even CTA's barriers
    const uint32_t tx = 2u * (uint32_t)stage_bytes;
    // Weight rows n .. of a tile in the image seen as one column of 64-value rows; a tile may end behind the last block: that block once
    // more, never stored.
    auto image_row = [&](int n) { return (min(n >> 7, p.n_blocks - 1) + (DUAL ? (int)rank * p.n_blocks : 0)) * p.k_blocks * 128 + (n & 127); };
    // 96 rows begin at a multiple of 32 and lie in one block or two: a box of 64 and one of 32, whichever comes first
    const bool split = !DUAL && p.bn == 192;
    int tm = 0, tn = 0, xr = 0, wr = 0, wr32 = 0, at64 = 0, at32 = 0;
    auto enter_tile = [&](int tile) {
      pair_tile_coords(p, tile, &tm, &tn);
      xr = (tm * 2 + (int)rank) * kPrBM;
      const int n = DUAL ? tn * 128 : tn * p.bn + (int)rank * w_rows;
      if (split) {
        at64 = n & 32;
        at32 = 64 - 2 * (n & 32);
        wr32 = image_row(n + at32);
      }
      wr = image_row(n + at64);
    };
    auto load_w = [&](int kb, int s) {
      uint8_t* dst = smem + s * stage_bytes + kPrPiece;
      pair_tma_load_2d(dst + at64 * 128, &tmW, full0 + s * 8, 0, wr + kb * 128);
      if (split) pair_tma_load_2d(dst + at32 * 128, &tmW32, full0 + s * 8, 0, wr32 + kb * 128);
    };
    if (total) enter_tile(first);
    // weights never depend on the kernel before this one: the first ring fill starts ahead of the dependency wait
    const int pre = min(min(p.stages, p.k_blocks), total);
    if (lead) {
      for (int i = 0; i < pre; ++i) {
        if (rank == 0) mbar_arrive_expect_tx(&ctl->full[i], tx);
        load_w(i, i);
      }
    }
    pdl_wait();
    if (lead)
      for (int i = 0; i < pre; ++i) pair_tma_load_2d(smem + i * stage_bytes, &tmA, full0 + i * 8, i * kPrBK, xr);
    int tile = first, kb = pre, s = pre == p.stages ? 0 : pre;
    uint32_t phase = pre == p.stages ? 0 : 1;              // a stage's first release completes phase 0; before it nothing is waited for
    bool go = true;
    for (int i = pre; i < total; ++i, ++kb) {
      if (kb == p.k_blocks) {
        kb = 0;
        tile += step;
        enter_tile(tile);
      }
      const bool free = wait(&ctl->empty[s], phase, kStatusTmaTimeout, i);
      if (free && lead) {
        if (rank == 0) mbar_arrive_expect_tx(&ctl->full[s], tx);
        load_w(kb, s);
        pair_tma_load_2d(smem + s * stage_bytes, &tmA, full0 + s * 8, kb * kPrBK, xr);
      }
      go = agreed(free);
      if (!go) break;
      if (++s == p.stages) { s = 0; phase ^= 1u; }
    }
    // The last stages' releases come from the even CTA's commits: neither CTA may leave before they are in.
    for (int i = max(0, total - p.stages); go && i < total; ++i) go = agreed(wait(&ctl->empty[i % p.stages], (uint32_t)(i / p.stages) & 1u, kStatusTmaTimeout, i));
  } else if (warp == 1) {
    // ------------------------------------------------- MMA issuer (even CTA) ----
    pdl_wait();
    if (rank == 0) {
      const bool lead = elect_one();
      const uint32_t idesc = umma_idesc_f16(2 * kPrBM, acc_cols, Num<T>::kFmt);
      // The issuing lane's own instructions bound the main loop if there are many of them: the stage counts up instead of being divided
      // out, the operand descriptors advance by constants (16-byte units).
      const uint64_t a_desc = umma_desc_k128(smem_u32(smem)), b_desc = umma_desc_k128(smem_u32(smem) + kPrPiece);
      const uint32_t stage_step = (uint32_t)(stage_bytes >> 4);
      int s = 0, lt = 0;
      uint32_t phase = 0, at = 0;
      for (int tile = first; tile < tiles; tile += step, ++lt) {
        const int b = lt & 1;
        if (!agreed(wait(&ctl->acc_empty[b], (((uint32_t)(lt >> 1)) & 1u) ^ 1u, kStatusMmaTimeout, lt) && limit)) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + (uint32_t)(b * 256);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          wait(&ctl->full[s], phase, kStatusMmaTimeout, lt);
          tc_fence_after_sync();
          if (lead) {
            const uint64_t ad = a_desc + at, bd = b_desc + at;
            pair_umma_f16(acc, ad, bd, idesc, kb ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < kPrBK / 16; ++k) pair_umma_f16(acc, ad + 2 * k, bd + 2 * k, idesc, 1u);
            if (limit) pair_umma_commit(&ctl->empty[s]);
          }
          at += stage_step;
          if (++s == p.stages) { s = 0; at = 0; phase ^= 1u; }
        }
        if (lead) pair_umma_commit(&ctl->acc_full[b]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue ----
    pdl_wait();
    const int ew = warp - 2, quarter = warp & 3, group = ew >> 2;      // a warp reads the tensor-memory lanes of its quarter
    const T* bias = EXTRA ? reinterpret_cast<const T*>(p.bias) : nullptr;
    const T* scale = EXTRA ? reinterpret_cast<const T*>(p.scale) : nullptr;
    const int out_cols = DUAL ? 128 : p.bn, chunks = out_cols / 64;
    uint8_t* stg = epi_stage + (size_t)ew * 2 * kPrChunk;
    const uint32_t acc_empty0 = dsmem_addr(smem_u32(&ctl->acc_empty[0]), 0);

    // The warp's chunks, tile after tile: every other one of a tile, the first of the pair's lt-th tile being group lt & 1's where a tile has
    // three.  `cur` is being finished, the residual and the column vectors of the one behind it are on their way.
    struct Chunk { int tile, c, col, row; };
    auto first_chunk = [&](int lt) { return chunks == 3 ? (group + lt) & 1 : group; };
    auto locate = [&](Chunk& k) {
      if (k.tile >= tiles) return;
      int tm, tn;
      pair_tile_coords(p, k.tile, &tm, &tn);
      k.col = tn * out_cols + k.c * 64;
      k.row = (tm * 2 + (int)rank) * kPrBM + quarter * 32;
    };
    auto live = [&](const Chunk& k) { return k.tile < tiles && k.row < p.M && k.col < p.N; };
    // Once a wait of this warp has run out, or another role has given up (limit == 0), the warp goes through its chunks without asking for a
    // residual, handing an accumulator back or storing.
    // Two columns to a lane, put together when they are used: an instruction on them here would wait for the trip to memory.
    struct Cols {
      uint16_t lo = 0, hi = 0;
      __device__ __forceinline__ uint32_t both() const { return (uint32_t)lo | ((uint32_t)hi << 16); }
    };
    struct Vecs { Cols bg, bu, sg, su; float rs; };
    auto pair_of = [&](const T* v, int n) -> Cols {
      Cols c;
      if (n < p.N) c.lo = *reinterpret_cast<const uint16_t*>(v + n);
      if (n + 1 < p.N) c.hi = *reinterpret_cast<const uint16_t*>(v + n + 1);
      return c;
    };
    auto ask = [&](const Chunk& k, int buf, Vecs& v) {
      v = {};
      v.rs = 1.f;
      if (!live(k)) return;
      if constexpr (EXTRA) {
        const int n = k.col + 2 * lane;
        if (bias) v.bg = pair_of(bias, n);
        if (scale) v.sg = pair_of(scale, n);
        if (DUAL && bias) v.bu = pair_of(bias + p.dual_offset, n);
        if (DUAL && scale) v.su = pair_of(scale + p.dual_offset, n);
        if (p.row_scale && k.row + lane < p.M) v.rs = p.row_scale[k.row + lane];
      }
      if (p.residual && lane == 0 && limit) {
        bulk_wait_read_all();                              // this buffer's last result has left
        mbar_arrive_expect_tx(&ctl->res[ew][buf], kPrChunk);
        tma_load_2d(stg + buf * kPrChunk, &tmR, &ctl->res[ew][buf], k.col, k.row);
      }
    };
    Chunk cur = {first, group, 0, 0};
    locate(cur);
    Vecs vec;
    uint32_t res_phase = 0;                                // bit b: parity that buffer b's next residual completes
    int buf = 0, lt = 0;
    ask(cur, 0, vec);
    for (int tile = first; tile < tiles; tile += step, ++lt) {
      const int b = lt & 1;
      wait(&ctl->acc_full[b], (uint32_t)(lt >> 1) & 1u, kStatusEpilogueTimeout, tile);
      if (*gave_up) limit = 0;
      tc_fence_after_sync();
      // The accumulator may be overwritten by the pair's tile after next once this warp's last values are in registers: the arrival is
      // remote for the odd CTA and its release would wait for the stores below.
      bool released = false;
      auto release = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0 && limit) mbar_arrive_cluster(acc_empty0 + b * 8);
        released = true;
      };
      while (cur.tile == tile) {
        Chunk next = cur;
        next.c += 2;
        if (next.c >= chunks) { next.c = first_chunk(lt + 1); next.tile += step; }
        locate(next);
        Vecs vnext;
        const bool now = live(cur);
        ask(next, now ? buf ^ 1 : buf, vnext);
        if (now) {
          uint8_t* tile_out = stg + buf * kPrChunk;
          if (p.residual) {
            wait(&ctl->res[ew][buf], (res_phase >> buf) & 1u, kStatusTmaTimeout, tile);
            res_phase ^= 1u << buf;
          } else if (lane == 0) {
            bulk_wait_read_1();
          }
          __syncwarp();
          const uint32_t bg = vec.bg.both(), bu = vec.bu.both(), sg = vec.sg.both(), su = vec.su.both();
          const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * 256 + cur.c * 64);
#pragma unroll
          for (int h = 0; h < 2; ++h) {                    // 32 columns per tensor-memory trip
            uint32_t ra[32], rb[DUAL ? 32 : 1];
            tmem_ld32(acc + h * 32, ra);
            if constexpr (DUAL) tmem_ld32(acc + 128 + h * 32, rb);
            tmem_ld_wait();
            if (h == 1 && next.tile != tile) release();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              float g[16], u[16], v[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                g[j] = __uint_as_float(ra[q * 16 + j]);
                u[j] = 0.f;
                if constexpr (DUAL) u[j] = __uint_as_float(rb[q * 16 + j]);
              }
              if constexpr (EXTRA) {
                if (p.row_scale) {
#pragma unroll
                  for (int j = 0; j < 16; ++j) { g[j] *= vec.rs; u[j] *= vec.rs; }
                }
                // One test for all columns: with one for each, every column's shuffle was waited for by itself.  3072 x 3840 x 1152 with a bias, us:
                // that and the vectors waited for where they are asked for 25.5, so 23.8 (no bias 23.1); 3072 x 4304 x 1152, bias and GELU 34.1 / 28.6
                // (24.7 without either).
                auto affine = [&](float (&x)[16], uint32_t sv, uint32_t bv) {
                  if (scale) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                      const uint32_t w = __shfl_sync(0xffffffffu, sv, h * 16 + q * 8 + j);
                      const float2 f = Num<T>::to_f2(*reinterpret_cast<const typename Num<T>::T2*>(&w));
                      x[2 * j] *= f.x;
                      x[2 * j + 1] *= f.y;
                    }
                  }
                  if (bias) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                      const uint32_t w = __shfl_sync(0xffffffffu, bv, h * 16 + q * 8 + j);
                      const float2 f = Num<T>::to_f2(*reinterpret_cast<const typename Num<T>::T2*>(&w));
                      x[2 * j] += f.x;
                      x[2 * j + 1] += f.y;
                    }
                  }
                };
                affine(g, sg, bg);
                if (DUAL) affine(u, su, bu);
              }
              apply_act_n<16>(p.act, g, u, v, p.act_args);
              // row `lane` of the staging tile, 128-byte swizzled as the bulk copies lay it out
#pragma unroll
              for (int o = 0; o < 2; ++o) {
                const int ch = h * 4 + q * 2 + o;
                T* at = reinterpret_cast<T*>(tile_out + lane * 128 + ((ch ^ (lane & 7)) << 4));
                float f[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = v[o * 8 + j];
                if (p.residual) {
                  float r[8];
                  unpack8<T>(*reinterpret_cast<const uint4*>(at), r);
#pragma unroll
                  for (int j = 0; j < 8; ++j) f[j] += r[j];
                }
                store8(at, f);
              }
            }
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0 && limit) {
            tma_store_2d(&tmO, tile_out, cur.col, cur.row);
            bulk_commit_group();
          }
          buf ^= 1;
        }
        cur = next;
        vec = vnext;
      }
      if (!released) release();                            // a last chunk without rows or columns
    }
    if (lane == 0) bulk_wait_all();                        // the last stores are complete before the CTA retires
  }
  __syncwarp();
  tc_fence_before_sync();
  cluster_sync_all();                                      // the even CTA's MMAs read the odd one's shared memory to the end
  if (*gave_up) settle_pair(&ctl->settled, rank, warp);
  if (warp == 1) pair_tmem_dealloc(tmem_base, 512u);
}

int ps_forced_band();                                            // gemm_ps.cu

template <typename T, bool DUAL, bool EXTRA>
static int launch_pair(const RfGemm* g, int bn, cudaStream_t stream) {
  auto kfn = gemm_pair_kernel<T, DUAL, EXTRA>;
  RF_ALLOW_SMEM_PER_DEVICE(kfn, 227 * 1024);
  GemmPairParams p = {};
  p.bias = g->bias; p.scale = g->scale; p.row_scale = g->row_scale; p.status = g->status;
  p.M = g->M; p.N = g->N; p.k_blocks = ceil_div(g->K, kPrBK); p.bn = bn;
  p.act = g->act; p.act_args = {g->act_limit, g->act_alpha}; p.dual_offset = g->dual_offset;
  p.n_blocks = ceil_div(g->N, 128);
  p.tiles_m = ceil_div(g->M, 2 * kPrBM); p.tiles_n = ceil_div(g->N, bn);
  p.residual = g->residual != nullptr;
  const int w_rows = DUAL ? 128 : bn / 2;
  CUtensorMap tmA, tmW, tmW32, tmO, tmR;
  int rc = make_tmap_2d(&tmA, g->x, g->dtype, 2, g->K, g->M, g->ldx, kPrBK, kPrBM, true);
  if (rc) return rc;
  // the weight image as one column of 64-value rows, already in the order that shared memory wants
  const uint64_t image_rows = (uint64_t)(DUAL ? 2 : 1) * p.n_blocks * p.k_blocks * 128;
  rc = make_tmap_2d(&tmW, g->w, g->dtype, 2, kPrBK, image_rows, kPrBK, kPrBK, w_rows == 96 ? 64 : w_rows, false);
  if (rc) return rc;
  tmW32 = tmW;
  if (w_rows == 96) {
    rc = make_tmap_2d(&tmW32, g->w, g->dtype, 2, kPrBK, image_rows, kPrBK, kPrBK, 32, false);
    if (rc) return rc;
  }
  rc = make_tmap_2d(&tmO, g->out, g->dtype, 2, g->N, g->M, g->ldo, 64, 32, true);
  if (rc) return rc;
  tmR = tmO;
  if (p.residual) {
    rc = make_tmap_2d(&tmR, g->residual, g->dtype, 2, g->N, g->M, g->ldr, 64, 32, true);
    if (rc) return rc;
  }
  // a band of activation rows of about 16 MB: it and a weight matrix of a few tens of MB stay in L2 together
  p.band = (int)std::max<int64_t>(1, std::min<int64_t>(p.tiles_m, (16ll << 20) / std::max<int64_t>(1, (int64_t)2 * kPrBM * g->K * 2)));
  if (ps_forced_band() > 0) p.band = std::min(p.tiles_m, ps_forced_band());
  const int stage_bytes = kPrPiece + w_rows * kPrBK * 2;
  const int other = (int)sizeof(GemmPairCtl) + 1024 /*alignment slack*/ + kPrEpiWarps * 2 * kPrChunk;
  p.stages = std::min(kPrMaxStages, (227 * 1024 - other) / stage_bytes);
  const size_t smem = (size_t)p.stages * stage_bytes + other;
  const int pairs = std::min(p.tiles_m * p.tiles_n, sm_count() / 2);
  RF_CUDA_CHECK(::rf::launch_clusters(kfn, dim3(2 * pairs), dim3(64 + 32 * kPrEpiWarps), smem, stream, dim3(2), tmA, tmW, tmW32, tmO, tmR, p));
  ::rf::count_launch();
  return RF_OK;
}

// What the kernel can do: tile-major 16-bit weights, results and residual that bulk tensor copies can write and read.
static bool pair_can(const RfGemm* g) {
  if (!g->w_packed || g->w_int8 || g->ar_world > 1 || g->ss_in || g->ss_out || g->mul || g->norm_x) return false;
  if ((g->ldo & 7) || (reinterpret_cast<uintptr_t>(g->out) & 15)) return false;
  if (g->residual && ((g->ldr & 7) || (reinterpret_cast<uintptr_t>(g->residual) & 15))) return false;
  return (reinterpret_cast<uintptr_t>(g->x) & 15) == 0;
}

// Tile width and estimated time.  A k block of a tile takes 205 ns at 128 columns, 270 at 192 and 345 at 256 with all SMs busy; tiles of few k
// blocks take what their epilogue does, longer with a residual and vectors to add.  Narrow tiles have less to fill and drain; 192 columns are for
// the sizes whose tiles otherwise leave SMs idle in the last round.  The constants are the best fit to 396 sizes (300 to 8192 rows, 18 weights, with
// and without a residual): the width taken is 0.5 % off the best one in the mean, 2.2 % without 192.  Measured, fp16, us, 128 / 192 / 256 columns
// (model): 825 x 2048 x 16384 56 / 67 / 81 (56 / 75 / 94), 1536 x 2048 x 16384 103 / 77 / 87 (109 / 75 / 94), 3072 x 1152 x 4304 29.7 / 24.1 / 28.4
// (32 / 24 / 29), 1536 x 8192 x 2048 42 / - / 38 (43 / 32 / 38), 825 x 1152 x 1152 7.3 / - / 10.6 (7.4 / 10 / 12).
struct PairShape { int bn; long ns; };
static PairShape pair_shape(const RfGemm* g) {
  const bool extra = g->bias || g->scale || g->row_scale || g->residual;
  const long k_blocks = ceil_div(g->K, kPrBK), pairs = std::max(1, sm_count() / 2);
  auto estimate = [&](int cols, long kb_ns, long around, long drain) {
    const long tiles = (long)ceil_div(g->M, 2 * kPrBM) * ceil_div(g->N, cols);
    return around + (tiles + pairs - 1) / pairs * std::max(k_blocks * kb_ns, drain);
  };
  if (g->dual_offset > 0) return {128, estimate(128, 345, extra ? 8300 : 5300, 2000)};
  const PairShape shapes[3] = {{128, estimate(128, 205, extra ? 5200 : 3700, extra ? 3100 : 1650)},
                               {192, estimate(192, 270, extra ? 8000 : 5500, extra ? 3800 : 1900)},
                               {256, estimate(256, 345, extra ? 8300 : 5300, extra ? 5000 : 2000)}};
  PairShape best = shapes[0];
  for (const PairShape& s : shapes)
    if (s.ns < best.ns) best = s;
  return best;
}

bool gemm_pairs_on();                                            // gemm_ps.cu

// Estimated time in ns where the kernel takes this GEMM, 0 where it cannot or may not.
long gemm_pair_ns(const RfGemm* g) { return gemm_pairs_on() && pair_can(g) ? pair_shape(g).ns : 0; }
// Columns of a tile (of a GLU pair: of its result)
int gemm_pair_cols(const RfGemm* g) { return pair_shape(g).bn; }

int launch_gemm_pair(const RfGemm* g, cudaStream_t stream) {
  const int bn = pair_shape(g).bn;
  const bool dual = g->dual_offset > 0, extra = g->bias || g->scale || g->row_scale;
#define RF_PAIR(T)                                                                                             \
  return dual ? (extra ? launch_pair<T, true, true>(g, bn, stream) : launch_pair<T, true, false>(g, bn, stream)) \
              : (extra ? launch_pair<T, false, true>(g, bn, stream) : launch_pair<T, false, false>(g, bn, stream))
  if (g->dtype == 0) { RF_PAIR(__half); }
  RF_PAIR(__nv_bfloat16);
#undef RF_PAIR
}

}  // namespace rf
