// GEMM of very few rows (at most 16) over tile-major weights:  out[M,N] = epilogue( x[M,K] . w[N,K]^T ).
//
// At these sizes the time is a pass over the weights plus what a launch adds around it, and the tcgen05 kernel (gemm_tc.cu) adds a lot:
// barriers, tensor-memory allocation, a ring whose stages are handed from warp to warp, and a cluster rendezvous on both sides of the split-K
// reduction.  Here every warp has a ring of its own and feeds its own MMAs.
//
//  * A CTA of eight warps takes strips of 16 output features (int8 also 32); its warps share a strip's 64-column k blocks.  Inside a block a lane
//    (g = lane / 4, t = lane % 4) holds 16 bytes of rows g and g + 8: eight values (16-bit), sixteen (int8) or, with 8 bytes, sixteen
//    (int4), all neighbours along k.  mma.sync does not care which k a slot stands for as long as both operands agree, so the lane's
//    words are the A fragments as they come, and the same k range of token g is the B fragment: no shuffles, and no meeting of warps.
//    int8 and int4 are widened in registers on the way.
//  * Four to eight blocks of weights per warp (two of a 16-bit and four of an int8 GLU pair; 64 KB a CTA, 40 of int4 and 70 to 80 of an
//    int4 pair; two CTAs an SM) are on their way in the warp's ring, over the ends of strips too; the
//    first ones are asked for ahead of the dependency wait.  cp.async, and not loads into registers: a warp waits for its loads on a handful of
//    counters, and with weights and x on the same ones every block waited for the newest (12 x 151936 x 4096 int8 215 us in registers, 160 now;
//    1 x 12288 x 4096 int8 SwiGLU 24.7 / 18.2).  Each lane copies what it will read; only int4 blocks, 512 bytes, are shared by the warp.
//  * x comes from L2 or L1, one block ahead; what the epilogue adds and multiplies by ahead of a strip's products.
//  * The warps' sums meet in shared memory once per strip; one thread finishes one value.
//  * A folded RMSNorm needs no sums of squares from the kernel before (norm_x): every CTA reads all of x anyway and squares it on the way.
//    GEMMs that are given sums (ss_in) run on gemm_tc.cu: adding them up here made the kernel slower without them (int8, 12 rows, 4 %).
//
// fp16, us, this kernel / gemm_tc.cu: 1 x 4096 x 1024 3.1 / 5.7, 1 x 1024 x 2048 3.0 / 5.5, 8 x 2048 x 2048 4.1 / 6.2, 1 x 6144 x 4096 10.5 / 12.9,
// 1 x 4096 x 12288 17.0 / 19.5, 16 x 3072 x 2048 5.1 / 6.6, 16 x 4096 x 4096 9.2 / 10.5; SwiGLU 1 x 12288 x 4096 31.5 / 35.3 (30.3 at the copy
// rate), 16 x 8192 x 2048 13.9 / 15.2.  int8: 1 x 4096 x 4096 6.3 / 11.9, 12 x 12288 x 4096 SwiGLU 24.0 / 44.4, 12 x 151936 x 4096 160 / 242; int4:
// 12 x 12288 x 4096 SwiGLU 31.7 / 52.8, 12 x 4096 x 12288 18.7 / 29.4.  (Row tiles that start their k blocks at different places, as gemm_tc.cu has
// them: up to a quarter slower.  The strips of a row tile then still share its blocks, but the blocks read side by side are no longer neighbours.)
#include "../common/dtype.cuh"
#include "../common/host_util.h"
#include "../common/mma.cuh"
#include "../common/ptx.cuh"
#include "../rf_api.h"

namespace rf {

constexpr int kRowsWarps = 8, kRowsStrip = 16, kRowsBK = 64;

struct GemmRowsParams {
  const void* x; int64_t ldx;
  void* out; int64_t ldo;
  const void* residual; int64_t ldr;
  const void* bias; const void* scale; const float* row_scale;
  const uint8_t* w;
  int M, N, K, k_blocks, strips, act, dual_offset, dual_tiles, blk_bytes;
  ActArgs act_args;
  int ns, fp4;                  // int4: scales per row of a block, e2m1 codes
  int norm;                     // scale every token by the reciprocal root mean square of its row of x
  float inv_dim, eps;
};

// weights are read once and never written while the library runs: around L1, and allowed ahead of the dependency wait
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds8(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint16_t lds2(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}

// Ring of a warp: `depth` blocks of weights, each `bytes` (of every accumulator) long: 16 rows of 64 columns, behind int4 up to four scales a row.
template <int BITS, bool DUAL, int NT, int SF> struct RowsRing {
  static constexpr int bytes = BITS == 16 ? 2048 : BITS == 8 ? 1024 : 512 + kRowsStrip * 8;
  // an int4 pair of 9 to 16 rows, whose sums take 34 KB: seven, so that a second CTA fits (fp16, us, with eight / seven: 12 x 12288 x 4096
  // SwiGLU, scales of 64 columns, 38.7 / 31.7, 16 x 9728 x 2560 23.3 / 17.4)
  static constexpr int depth = (DUAL ? (BITS == 16 ? 2 : BITS == 8 ? 4 : NT == 1 ? 8 : 7) : (BITS == 16 ? 4 : 8)) / SF;
  static constexpr int slot_bytes = bytes * SF * (DUAL ? 2 : 1), warp_bytes = depth * slot_bytes;
  static constexpr int total = warp_bytes * kRowsWarps;
};

// SF: groups of 16 features in a strip
template <typename T, int BITS, bool DUAL, int NT, int SF>
__global__ void __launch_bounds__(kRowsWarps * 32, 2)
gemm_rows_kernel(const GemmRowsParams p) {
  using Ring = RowsRing<BITS, DUAL, NT, SF>;
  constexpr int kAcc = DUAL ? 2 : 1, kStrip = kRowsStrip * SF;
  constexpr int kPitch = kStrip + 1, kSumBufs = SF == 1 ? 2 : 1;
  extern __shared__ __align__(128) uint8_t ring_mem[];
  __shared__ float sums[kSumBufs][kRowsWarps][kAcc][NT * 8][kPitch];
  __shared__ float squares[kRowsWarps][NT * 8];
  __shared__ float rstd[NT * 8];
  static_assert(2 * (Ring::total + sizeof(sums) + sizeof(squares) + sizeof(rstd) + 1024) <= 228 * 1024, "two CTAs have to fit an SM");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int KB = p.k_blocks, nk = (KB - warp + kRowsWarps - 1) / kRowsWarps;      // this warp's blocks of a strip: warp, warp + 8, ...
  const uint32_t ring = smem_u32(ring_mem) + warp * Ring::warp_bytes;
  pdl_launch_dependents();

  // the next block to ask for: block aj of strip `as`, into slot `aslot`; one group per call, also behind the last block
  int as = blockIdx.x, aj = 0, aslot = 0;
  auto ask = [&] {
    if (nk > 0 && as < p.strips) {
      const int rt = as / (8 / SF), strip0 = (as % (8 / SF)) * kStrip;      // 128-row tile, first row inside it
#pragma unroll
      for (int cf = 0; cf < kAcc * SF; ++cf) {
        const int c = cf / SF, r0 = strip0 + cf % SF * kRowsStrip;
        const uint8_t* blk = p.w + ((size_t)(rt + c * p.dual_tiles) * KB + warp + aj * kRowsWarps) * p.blk_bytes;
        const uint32_t dst = ring + (uint32_t)(aslot * Ring::slot_bytes + cf * Ring::bytes + lane * 16);
        if constexpr (BITS == 16) {                                 // a lane copies what it will read: 16-byte pieces t and 4 + t of rows g and g + 8
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint8_t* row = blk + (r0 + g + 8 * h) * 128;      // swizzled by row % 8 == g
            copy16(dst + (0 + h) * 512, row + ((t ^ g) << 4));
            copy16(dst + (2 + h) * 512, row + (((4 + t) ^ g) << 4));
          }
        } else if constexpr (BITS == 8) {                           // here too: lane 4 g + t has 16 values of rows g and g + 8
          copy16(dst, blk + r0 * 64 + lane * 16);
          copy16(dst + 512, blk + r0 * 64 + 512 + lane * 16);
        } else {
          copy16(dst, blk + r0 * 32 + lane * 16);
          if (lane < 2 * p.ns) copy16(dst + 512, blk + 4096 + r0 * p.ns * 2 + lane * 16);
        }
      }
      if (++aj == nk) { aj = 0; as += gridDim.x; }
      if (++aslot == Ring::depth) aslot = 0;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int u = 0; u < Ring::depth; ++u) ask();
  pdl_wait();

  // x of a block: 16 values of token g of every group of eight, in two 16-byte pieces that match the weights' k order
  const T* x = reinterpret_cast<const T*>(p.x);
  uint4 xn[NT][2];
  auto load_x = [&](int j) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int tok = n * 8 + g;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = (warp + j * kRowsWarps) * kRowsBK + (BITS == 16 ? (h * 4 + t) * 8 : t * 16 + h * 8);
        xn[n][h] = make_uint4(0u, 0u, 0u, 0u);
        if (tok < p.M && k < p.K) xn[n][h] = *reinterpret_cast<const uint4*>(x + (size_t)tok * p.ldx + k);
      }
    }
  };
  if (nk > 0) load_x(0);
  const int tok = tid >> 4, r = tid & 15;        // the value that this thread finishes in every group of 16 features
  const T* bias = reinterpret_cast<const T*>(p.bias);
  const T* scale = reinterpret_cast<const T*>(p.scale);
  const T* resid = reinterpret_cast<const T*>(p.residual);
  const float row_scale = p.row_scale && tok < p.M ? p.row_scale[tok] : 1.f;
  float sq[NT] = {};
  int buf = 0, slot = 0;
  for (int strip = blockIdx.x; strip < p.strips; strip += gridDim.x, buf ^= 1) {
    const bool first = strip == (int)blockIdx.x;
    // what the epilogue adds and multiplies by is asked for ahead of the products
    const T one = Num<T>::from_f(1.f), zero = Num<T>::from_f(0.f);
    T sc[SF][2], bi[SF][2], re[SF];
#pragma unroll
    for (int f = 0; f < SF; ++f) {
      const int n_out = strip * kStrip + f * kRowsStrip + r;
      sc[f][0] = sc[f][1] = one;
      bi[f][0] = bi[f][1] = re[f] = zero;
      if (tok >= p.M || n_out >= p.N) continue;
      if (scale) { sc[f][0] = scale[n_out]; if (DUAL) sc[f][1] = scale[p.dual_offset + n_out]; }
      if (bias) { bi[f][0] = bias[n_out]; if (DUAL) bi[f][1] = bias[p.dual_offset + n_out]; }
      if (resid) re[f] = resid[(size_t)tok * p.ldr + n_out];
    }
    float acc[kAcc * SF][NT][4] = {};
    for (int j = 0; j < nk; ++j) {
      uint4 b[NT][2];
#pragma unroll
      for (int n = 0; n < NT; ++n) { b[n][0] = xn[n][0]; b[n][1] = xn[n][1]; }
      load_x(j + 1 < nk ? j + 1 : 0);            // x is the same for every strip
      asm volatile("cp.async.wait_group %0;" ::"n"(Ring::depth - 1) : "memory");
      if constexpr (BITS == 4) __syncwarp();     // its pieces were copied by other lanes
      if (p.norm && first) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float f[8];
            unpack8<T>(b[n][h], f);
#pragma unroll
            for (int i = 0; i < 8; ++i) sq[n] = fmaf(f[i], f[i], sq[n]);
          }
      }
#pragma unroll
      for (int c = 0; c < kAcc * SF; ++c) {
        const uint32_t src = ring + (uint32_t)(slot * Ring::slot_bytes + c * Ring::bytes);
        uint4 q[2];
        uint2 q4[2];
        if constexpr (BITS == 8) { q[0] = lds16(src + lane * 16); q[1] = lds16(src + 512 + lane * 16); }
        if constexpr (BITS == 4) { q4[0] = lds8(src + lane * 8); q4[1] = lds8(src + 256 + lane * 8); }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 lo, hi;                                             // eight values along k of row g, of row g + 8
          if constexpr (BITS == 16) {
            lo = lds16(src + (2 * h) * 512 + lane * 16);
            hi = lds16(src + (2 * h + 1) * 512 + lane * 16);
          } else if constexpr (BITS == 8) {
            lo = widen_i8x8<T>(h ? make_uint2(q[0].z, q[0].w) : make_uint2(q[0].x, q[0].y));
            hi = widen_i8x8<T>(h ? make_uint2(q[1].z, q[1].w) : make_uint2(q[1].x, q[1].y));
          } else {
            T s[2] = {one, one};                                    // word w of a row covers columns 8 w .. 8 w + 7
            if (p.ns) {
#pragma unroll
              for (int row = 0; row < 2; ++row) {
                const uint16_t bits = lds2(src + 512 + (uint32_t)((g + 8 * row) * p.ns + ((2 * t + h) * p.ns >> 3)) * 2);
                s[row] = *reinterpret_cast<const T*>(&bits);
              }
            }
            const uint32_t w0 = h ? q4[0].y : q4[0].x, w1 = h ? q4[1].y : q4[1].x;
            lo = p.fp4 ? widen_e2m1x8<T>(w0, s[0]) : widen_i4x8<T>(w0, s[0]);
            hi = p.fp4 ? widen_e2m1x8<T>(w1, s[1]) : widen_i4x8<T>(w1, s[1]);
          }
          const uint32_t a01[4] = {lo.x, hi.x, lo.y, hi.y}, a23[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            MmaOp<T>::mma(acc[c][n], a01, b[n][h].x, b[n][h].y);
            MmaOp<T>::mma(acc[c][n], a23, b[n][h].z, b[n][h].w);
          }
        }
      }
      if constexpr (BITS == 4) __syncwarp();
      ask();                                     // into the slot just read
      if (++slot == Ring::depth) slot = 0;
    }
    // ---- the warps' sums: token rows of 16 features; two buffers, so one rendezvous per strip is enough
    if constexpr (SF > 1) {
      if (!first) __syncthreads();               // one buffer: the strip before has been read
    }
#pragma unroll
    for (int c = 0; c < kAcc * SF; ++c)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          sums[kSumBufs == 2 ? buf : 0][warp][c / SF][n * 8 + 2 * t + (i & 1)][c % SF * kRowsStrip + g + 8 * (i >> 1)] = acc[c][n][i];
    if (p.norm && first) {
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        sq[n] += __shfl_xor_sync(0xffffffffu, sq[n], 1);
        sq[n] += __shfl_xor_sync(0xffffffffu, sq[n], 2);
        if (t == 0) squares[warp][n * 8 + g] = sq[n];
      }
    }
    __syncthreads();
    if (p.norm && first) {
      if (tid < NT * 8) {
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < kRowsWarps; ++i) v += squares[i][tid];
        rstd[tid] = rsqrtf(v * p.inv_dim + p.eps);
      }
      __syncthreads();
    }
#pragma unroll
    for (int f = 0; f < SF; ++f) {
      const int n_out = strip * kStrip + f * kRowsStrip + r;
      if (tok >= p.M || n_out >= p.N) continue;
      float gate = 0.f, up = 0.f;
#pragma unroll
      for (int w = 0; w < kRowsWarps; ++w) {
        gate += sums[kSumBufs == 2 ? buf : 0][w][0][tok][f * kRowsStrip + r];
        if (DUAL) up += sums[kSumBufs == 2 ? buf : 0][w][kAcc - 1][tok][f * kRowsStrip + r];
      }
      const float rs = p.norm ? rstd[tok] * row_scale : row_scale;
      gate *= rs;
      up *= rs;
      if (scale) { gate *= Num<T>::to_f(sc[f][0]); up *= Num<T>::to_f(sc[f][1]); }
      if (bias) { gate += Num<T>::to_f(bi[f][0]); up += Num<T>::to_f(bi[f][1]); }
      float v = apply_act(p.act, gate, up, p.act_args);
      if (resid) v += Num<T>::to_f(re[f]);
      reinterpret_cast<T*>(p.out)[(size_t)tok * p.ldo + n_out] = Num<T>::from_f(v);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ------------------------------------------------------------------ host side ----
static int rows_limit() {
  static const int v = [] { const char* e = getenv("RF_GEMM_ROWS"); return e ? atoi(e) : -1; }();
  return v >= 0 ? std::min(v, 16) : 16;
}

// Shapes this kernel takes.  Quantised weights, widened in registers instead of through the warps of another kernel, and GLU pairs win at every size
// (fp16, us, this kernel / gemm_tc.cu: 16 x 12288 x 4096 SwiGLU 35.4 / 35.9, 16 x 9728 x 2560 21.7 / 22.3).  Up to 8 rows what it pays is x, which
// every CTA reads, on long rows (8 x 2560 x 9728 13.3 / 14.0, 4 x 4096 x 12288 19.0 / 19.8, 8 x 4096 x 12288 20.8 / 20.0).  With 9 to 16 rows the
// products are twice as many, and long rows and an uneven last round of strips lose (16 x 4096 x 4096 9.2 / 10.5, 16 x 2560 x 4096 8.0 / 8.7;
// 16 x 6144 x 4096 14.7 / 13.5, 16 x 6144 x 2560 10.5 / 9.8, 16 x 2048 x 8192 12.2 / 11.7).
bool gemm_rows_takes(const RfGemm* g) {
  if (g->M > rows_limit() || !g->w_packed || g->ar_world > 1 || g->streaming_only == 2 || g->ss_in || g->ss_out || g->mul || g->force_splits || g->force_bn || g->force_swap >= 0)
    return false;
  if ((reinterpret_cast<uintptr_t>(g->x) & 15) != 0) return false;
  if (g->w_int8) return true;
  if (g->dual_offset > 0) return true;
  if (g->M <= 8) return (int64_t)g->M * g->K <= (80 << 10);
  return (int64_t)g->N * g->K <= (8 << 20) || (g->K <= 4096 && g->N <= 2 * kRowsStrip * sm_count());
}

template <typename T, int BITS, bool DUAL, int NT, int SF>
static int launch_rows_sf(const RfGemm* g, cudaStream_t stream) {
  auto kfn = gemm_rows_kernel<T, BITS, DUAL, NT, SF>;
  GemmRowsParams p = {};
  p.x = g->x; p.ldx = g->ldx; p.out = g->out; p.ldo = g->ldo; p.residual = g->residual; p.ldr = g->ldr;
  p.bias = g->bias; p.scale = g->scale; p.row_scale = g->row_scale;
  p.w = reinterpret_cast<const uint8_t*>(g->w);
  p.M = g->M; p.N = g->N; p.K = g->K; p.k_blocks = ceil_div(g->K, kRowsBK); p.strips = ceil_div(g->N, kRowsStrip * SF);
  p.act = g->act; p.act_args = {g->act_limit, g->act_alpha}; p.dual_offset = g->dual_offset; p.dual_tiles = ceil_div(g->N, 128);
  p.blk_bytes = BITS == 16 ? 16384 : BITS == 8 ? 8192 : rf_w4_block_bytes(g->w_group);
  p.ns = BITS == 4 && g->w_group > 0 ? kRowsBK / std::min(g->w_group, kRowsBK) : 0;
  p.fp4 = g->w_fp4;
  p.norm = g->norm_x;
  p.inv_dim = g->ss_dim > 0 ? 1.f / (float)g->ss_dim : 0.f;
  p.eps = g->ss_eps;
  constexpr int smem = RowsRing<BITS, DUAL, NT, SF>::total;
  RF_ALLOW_SMEM_PER_DEVICE(kfn, smem);
  RF_CUDA_CHECK(::rf::launch_k(kfn, dim3(std::min(p.strips, 2 * sm_count())), dim3(kRowsWarps * 32), smem, stream, 1, p));
  ::rf::count_launch();
  return RF_OK;
}

template <typename T, int BITS, bool DUAL, int NT>
static int launch_rows(const RfGemm* g, cudaStream_t stream) {
  // Strips of 32 features read x half as often, which with int8 weights is as many bytes as the weights themselves, as long as there is one for every SM.
  // int8, fp16, us, 16 / 32: 1 x 151936 x 4096 118 / 94 (the copy rate), 12 rows 167 / 126, 1 x 6144 x 4096 9.9 / 7.8, 12 rows 12.2 / 9.5, 8 x 9728 x 2048
  // 9.5 / 7.5; 1 x 4096 x 4096 6.2 / 6.9, 12 x 4096 x 12288 17.0 / 21.5.  Not GLU pairs, whose ring gets too short (12 x 12288 x 4096 24.5 / 27.4), nor
  // 16-bit weights (1 x 9728 x 2048 9.5 / 10.7).
  if constexpr (BITS == 8 && !DUAL) {
    if (ceil_div(g->N, 2 * kRowsStrip) > sm_count()) return launch_rows_sf<T, BITS, DUAL, NT, 2>(g, stream);
  }
  return launch_rows_sf<T, BITS, DUAL, NT, 1>(g, stream);
}

template <typename T, int BITS, int NT>
static int launch_rows_d(const RfGemm* g, cudaStream_t stream) {
  return g->dual_offset > 0 ? launch_rows<T, BITS, true, NT>(g, stream) : launch_rows<T, BITS, false, NT>(g, stream);
}

template <typename T>
static int launch_rows_t(const RfGemm* g, cudaStream_t stream) {
  if (g->w_bits == 4) return g->M <= 8 ? launch_rows_d<T, 4, 1>(g, stream) : launch_rows_d<T, 4, 2>(g, stream);
  if (g->w_int8) return g->M <= 8 ? launch_rows_d<T, 8, 1>(g, stream) : launch_rows_d<T, 8, 2>(g, stream);
  return g->M <= 8 ? launch_rows_d<T, 16, 1>(g, stream) : launch_rows_d<T, 16, 2>(g, stream);
}

int launch_gemm_rows(const RfGemm* g, cudaStream_t stream) {
  return g->dtype == 0 ? launch_rows_t<__half>(g, stream) : launch_rows_t<__nv_bfloat16>(g, stream);
}

}  // namespace rf
