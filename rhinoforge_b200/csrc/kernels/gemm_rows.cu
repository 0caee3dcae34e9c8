// GEMM of very few rows (at most 16) over tile-major weights:  out[M,N] = epilogue( x[M,K] . w[N,K]^T ).
//
// At these sizes the time is a pass over the weights plus what a launch adds around it, and the tcgen05 kernel (gemm_tc.cu) adds a lot:
// barriers, tensor-memory allocation, a ring through shared memory, and a cluster rendezvous on both sides of the split-K reduction.
// Here a weight goes from memory into the registers that feed the MMA and nowhere else.
//
//  * A CTA of eight warps takes strips of 16 output features; its warps share a strip's 64-column k blocks.  Inside a block a lane
//    (g = lane / 4, t = lane % 4) loads 16 bytes of rows g and g + 8: eight values (16-bit), sixteen (int8) or, with 8 bytes, sixteen
//    (int4), all neighbours along k.  mma.sync does not care which k a slot stands for as long as both operands agree, so the lane's
//    words are the A fragments as they come, and the same k range of token g is the B fragment: no shared memory, no shuffles.
//    int8 and int4 are widened in registers on the way.
//  * Two to four blocks of weights per warp are always on their way, over the ends of strips too; the first ones are asked for ahead of
//    the dependency wait.  x comes from L2 or L1, one block ahead.
//  * The warps' sums meet in shared memory once per strip; one thread finishes one value.
//  * A folded RMSNorm needs no sums of squares from the kernel before: every CTA reads all of x anyway and squares it on the way.
//
// fp16, us, this kernel / gemm_tc.cu: 1 x 4096 x 1024 3.1 / 5.7, 1 x 1024 x 2048 2.9 / 5.5, 8 x 2048 x 2048 3.7 / 6.2, 16 x 3072 x 2048 5.0 / 6.5,
// 1 x 4096 x 4096 8.0 / 10.0, 8 x 8192 x 2048 SwiGLU 13.0 / 15.1; not taken: 1 x 2048 x 8192 13.0 / 11.2, 1 x 6144 x 4096 14.3 / 13.0,
// 16 x 8192 x 2048 SwiGLU 16.3 / 15.3.  int8: 1 x 4096 x 4096 6.6 / 11.9, 12 x 12288 x 4096 SwiGLU 26.8 / 44.4, 12 x 151936 x 4096 215 / 242;
// int4: 12 x 12288 x 4096 SwiGLU 40.4 / 52.8.  (Row tiles that start their k blocks at different places, as gemm_tc.cu has them: up to a quarter
// slower.  The strips of a row tile then still share its blocks, but the blocks that are read side by side are no longer neighbours.)
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
__device__ __forceinline__ uint4 ldw16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ldw8(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// What a lane holds of one k block of a strip: rows g and g + 8.
template <int BITS> struct RowsA;
template <> struct RowsA<16> { uint4 q[2][2]; };                    // [32-column half][row]
template <> struct RowsA<8> { uint4 q[2]; };                        // [row]
template <> struct RowsA<4> { uint2 q[2]; uint32_t s[2]; };         // [row]; s: scales of the two words, 16 bits each

template <typename T, int BITS, bool DUAL, int NT>
__global__ void __launch_bounds__(kRowsWarps * 32, 2)
gemm_rows_kernel(const GemmRowsParams p) {
  constexpr int kAcc = DUAL ? 2 : 1;
  // Blocks of weights on their way per warp (2 KB of 16-bit values, 1 KB of int8, 0.5 KB of int4 each and accumulator).  x comes one block ahead
  // and not with its weights: a warp waits for its loads on a handful of counters, and with x four blocks ahead as well, blocks began to wait for
  // one another's (12 x 12288 x 4096 int8 SwiGLU 26.8 -> 33.3 us).
  constexpr int U = BITS == 16 && DUAL ? 2 : 4;                     // even: the x ring of two turns with it
  constexpr int kPitch = kRowsStrip + 1;
  __shared__ float sums[2][kRowsWarps][kAcc][NT * 8][kPitch];
  __shared__ float squares[kRowsWarps][NT * 8];
  __shared__ float rstd[NT * 8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int KB = p.k_blocks, nk = (KB - warp + kRowsWarps - 1) / kRowsWarps;      // this warp's blocks of a strip: warp, warp + 8, ...
  const int turns = (nk + U - 1) / U * U;                           // ... rounded up to whole turns of the ring
  pdl_launch_dependents();

  RowsA<BITS> a[U][kAcc];
  // asks for block j of a strip, or past the strip's last turn for one of this CTA's next strip
  auto ask = [&](RowsA<BITS> (&d)[kAcc], int strip, int j) {
    if (j >= turns) { j -= turns; strip += gridDim.x; }
    if (j >= nk || strip >= p.strips) return;
    const int rt = strip >> 3, r0 = (strip & 7) * kRowsStrip;       // 128-row tile, first row inside it
#pragma unroll
    for (int c = 0; c < kAcc; ++c) {
      const uint8_t* blk = p.w + ((size_t)(rt + c * p.dual_tiles) * KB + warp + j * kRowsWarps) * p.blk_bytes;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + g + 8 * h;                               // r % 8 == g: the swizzle of 16-bit rows
        if constexpr (BITS == 16) {
          d[c].q[0][h] = ldw16(blk + r * 128 + ((t ^ g) << 4));
          d[c].q[1][h] = ldw16(blk + r * 128 + (((4 + t) ^ g) << 4));
        } else if constexpr (BITS == 8) {
          d[c].q[h] = ldw16(blk + r * 64 + t * 16);
        } else {
          d[c].q[h] = ldw8(blk + r * 32 + t * 8);
          const T* sr = reinterpret_cast<const T*>(blk + 4096) + r * p.ns;         // word w covers columns 8 w .. 8 w + 7
          const T one = Num<T>::from_f(1.f);
          const T s0 = p.ns ? sr[(2 * t) * p.ns >> 3] : one, s1 = p.ns ? sr[(2 * t + 1) * p.ns >> 3] : one;
          d[c].s[h] = (uint32_t)*reinterpret_cast<const uint16_t*>(&s0) | ((uint32_t)*reinterpret_cast<const uint16_t*>(&s1) << 16);
        }
      }
    }
  };
  if (nk > 0) {
#pragma unroll
    for (int u = 0; u < U; ++u) ask(a[u], blockIdx.x, u);
  }
  pdl_wait();

  // x of a block: 16 values of token g of every group of eight, in two 16-byte pieces that match the weights' k order
  const T* x = reinterpret_cast<const T*>(p.x);
  uint4 xb[2][NT][2];
  auto load_x = [&](int j, uint4 (&d)[NT][2]) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int tok = n * 8 + g;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = (warp + j * kRowsWarps) * kRowsBK + (BITS == 16 ? (h * 4 + t) * 8 : t * 16 + h * 8);
        d[n][h] = make_uint4(0u, 0u, 0u, 0u);
        if (tok < p.M && k < p.K) d[n][h] = *reinterpret_cast<const uint4*>(x + (size_t)tok * p.ldx + k);
      }
    }
  };
  float sq[NT] = {};
  int buf = 0;
  for (int strip = blockIdx.x; strip < p.strips; strip += gridDim.x, buf ^= 1) {
    const bool first = strip == (int)blockIdx.x;
    float acc[kAcc][NT][4] = {};
    if (nk > 0) load_x(0, xb[0]);
    for (int j = 0; j < turns; j += U) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j + u < nk) {
          if (j + u + 1 < nk) load_x(j + u + 1, xb[(u + 1) & 1]);
          const auto& b = xb[u & 1];
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
          const RowsA<BITS> (&w)[kAcc] = a[u];
#pragma unroll
          for (int c = 0; c < kAcc; ++c) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint4 lo, hi;                                         // eight values along k of row g, of row g + 8
              if constexpr (BITS == 16) {
                lo = w[c].q[h][0];
                hi = w[c].q[h][1];
              } else if constexpr (BITS == 8) {
                lo = widen_i8x8<T>(h ? make_uint2(w[c].q[0].z, w[c].q[0].w) : make_uint2(w[c].q[0].x, w[c].q[0].y));
                hi = widen_i8x8<T>(h ? make_uint2(w[c].q[1].z, w[c].q[1].w) : make_uint2(w[c].q[1].x, w[c].q[1].y));
              } else {
                const uint16_t s0 = (uint16_t)(w[c].s[0] >> (16 * h)), s1 = (uint16_t)(w[c].s[1] >> (16 * h));
                const T t0 = *reinterpret_cast<const T*>(&s0), t1 = *reinterpret_cast<const T*>(&s1);
                const uint32_t q0 = h ? w[c].q[0].y : w[c].q[0].x, q1 = h ? w[c].q[1].y : w[c].q[1].x;
                lo = p.fp4 ? widen_e2m1x8<T>(q0, t0) : widen_i4x8<T>(q0, t0);
                hi = p.fp4 ? widen_e2m1x8<T>(q1, t1) : widen_i4x8<T>(q1, t1);
              }
              const uint32_t a01[4] = {lo.x, hi.x, lo.y, hi.y}, a23[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
              for (int n = 0; n < NT; ++n) {
                MmaOp<T>::mma(acc[c][n], a01, b[n][h].x, b[n][h].y);
                MmaOp<T>::mma(acc[c][n], a23, b[n][h].z, b[n][h].w);
              }
            }
          }
        }
        ask(a[u], strip, j + u + U);
      }
    }
    // ---- the warps' sums: token rows of 16 features; two buffers, so one rendezvous per strip is enough
#pragma unroll
    for (int c = 0; c < kAcc; ++c)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sums[buf][warp][c][n * 8 + 2 * t + (i & 1)][g + 8 * (i >> 1)] = acc[c][n][i];
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
    const T* bias = reinterpret_cast<const T*>(p.bias);
    const T* scale = reinterpret_cast<const T*>(p.scale);
    const T* resid = reinterpret_cast<const T*>(p.residual);
    for (int i = tid; i < p.M * kRowsStrip; i += kRowsWarps * 32) {
      const int tok = i >> 4, r = i & 15, n = strip * kRowsStrip + r;
      if (n >= p.N) continue;
      float gate = 0.f, up = 0.f;
#pragma unroll
      for (int w = 0; w < kRowsWarps; ++w) {
        gate += sums[buf][w][0][tok][r];
        if (DUAL) up += sums[buf][w][kAcc - 1][tok][r];
      }
      float rs = p.norm ? rstd[tok] : 1.f;
      if (p.row_scale) rs *= p.row_scale[tok];
      gate *= rs;
      up *= rs;
      if (scale) {
        gate *= Num<T>::to_f(scale[n]);
        if (DUAL) up *= Num<T>::to_f(scale[p.dual_offset + n]);
      }
      if (bias) {
        gate += Num<T>::to_f(bias[n]);
        if (DUAL) up += Num<T>::to_f(bias[p.dual_offset + n]);
      }
      float v = apply_act(p.act, gate, up, p.act_args);
      if (resid) v += Num<T>::to_f(resid[(size_t)tok * p.ldr + n]);
      reinterpret_cast<T*>(p.out)[(size_t)tok * p.ldo + n] = Num<T>::from_f(v);
    }
  }
}

// ------------------------------------------------------------------ host side ----
static int rows_limit() {
  static const int v = [] { const char* e = getenv("RF_GEMM_ROWS"); return e ? atoi(e) : -1; }();
  return v >= 0 ? std::min(v, 16) : 16;
}

// Shapes this kernel takes: see the table at the top of the file.  What it saves is the fixed part of a launch; what it pays are an uneven last
// round (a third more strips than places) and long walks along K by few warps.  Quantised weights, widened in registers instead of through
// shared memory, win at every size.
bool gemm_rows_takes(const RfGemm* g) {
  if (g->M > rows_limit() || !g->w_packed || g->ar_world > 1 || g->streaming_only == 2 || g->ss_out || g->mul || g->force_splits || g->force_bn || g->force_swap >= 0)
    return false;
  if ((reinterpret_cast<uintptr_t>(g->x) & 15) != 0) return false;
  if (g->w_int8) return true;
  const bool dual = g->dual_offset > 0;
  const int64_t values = (int64_t)g->N * g->K * (dual ? 2 : 1);
  return values <= (8 << 20) || (g->K <= 4096 && g->N <= 2 * kRowsStrip * sm_count() && !dual) || (dual && g->M <= 8 && g->K <= (g->M <= 2 ? 4096 : 2048));
}

template <typename T, int BITS, bool DUAL, int NT>
static int launch_rows(const RfGemm* g, cudaStream_t stream) {
  auto kfn = gemm_rows_kernel<T, BITS, DUAL, NT>;
  GemmRowsParams p = {};
  p.x = g->x; p.ldx = g->ldx; p.out = g->out; p.ldo = g->ldo; p.residual = g->residual; p.ldr = g->ldr;
  p.bias = g->bias; p.scale = g->scale; p.row_scale = g->row_scale;
  p.w = reinterpret_cast<const uint8_t*>(g->w);
  p.M = g->M; p.N = g->N; p.K = g->K; p.k_blocks = ceil_div(g->K, kRowsBK); p.strips = ceil_div(g->N, kRowsStrip);
  p.act = g->act; p.act_args = {g->act_limit, g->act_alpha}; p.dual_offset = g->dual_offset; p.dual_tiles = ceil_div(g->N, 128);
  p.blk_bytes = BITS == 16 ? 16384 : BITS == 8 ? 8192 : rf_w4_block_bytes(g->w_group);
  p.ns = BITS == 4 && g->w_group > 0 ? kRowsBK / std::min(g->w_group, kRowsBK) : 0;
  p.fp4 = g->w_fp4;
  p.norm = g->ss_in != nullptr;
  p.inv_dim = g->ss_dim > 0 ? 1.f / (float)g->ss_dim : 0.f;
  p.eps = g->ss_eps;
  RF_CUDA_CHECK(::rf::launch_k(kfn, dim3(std::min(p.strips, 2 * sm_count())), dim3(kRowsWarps * 32), 0, stream, 1, p));
  ::rf::count_launch();
  return RF_OK;
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
