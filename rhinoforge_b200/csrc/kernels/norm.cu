// Row normalisation kernels: RMSNorm (Qwen/Llama and Gemma "(1+w)" flavours,
// optional fused residual add, optional adaRMS scale/shift), LayerNorm, L2 norm.
// Replaces the reference's llama_rms_norm*, layer_norm* and l2norm operators
// (src/ops/rpu_rmsnorm.cpp, src/ops/rpu_layernorm.cpp, src/ops/rpu_l2norm.cpp)
// and the adaRMS SUB/MUL/ADD chain (src/fused/rpu_pi05_denoise_step_model.cpp:848-857).
#include <type_traits>

#include "../common/dtype.cuh"
#include "../common/host_util.h"
#include "../common/ptx.cuh"
#include "../rf_api.h"

namespace rf {

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

// Eight values of a row off its 16-byte boundary, or of one that may be.
template <typename T>
__device__ __forceinline__ void load8_at(const T* p, int whole, float (&f)[8]) {
  unpack8<T>(load_raw8(p, whole != 0), f);
}

// y = norm(x [+ residual]) ; if residual_out: residual_out = x + residual.
// mode bit0: gemma style weight (1 + w), product rounded once
// mod (optional, adaRMS): per-token [rows / rows_per_mod, 3H] = [scale | shift | gate];
//   y = norm(x) * (1 + scale) + shift   (weight is ignored when mod != null)
template <typename T>
__global__ void rmsnorm_kernel(const T* __restrict__ x, const T* __restrict__ residual,
                               const T* __restrict__ w, T* __restrict__ y,
                               T* __restrict__ residual_out, const T* __restrict__ mod,
                               int rows_per_mod, int H, int64_t ldx, int64_t ldy, float eps,
                               int mode, int whole) {
  pdl_prologue();
  extern __shared__ float srow[];  // H floats + 32
  float* red = srow + H;
  const int row = blockIdx.x;
  const T* xr = x + (size_t)row * ldx;
  const T* rr = residual ? residual + (size_t)row * ldx : nullptr;
  float ss = 0.f;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    float f[8];
    load8_at(xr + i, whole, f);
    if (rr) {
      float r[8];
      load8_at(rr + i, whole, r);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = Num<T>::to_f(Num<T>::from_f(f[j] + r[j]));
      if (residual_out) store8(residual_out + (size_t)row * ldx + i, f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      srow[i + j] = f[j];
      ss += f[j] * f[j];
    }
  }
  const float tot = block_sum(ss, red);
  const float rstd = rsqrtf(tot / (float)H + eps);
  const T* mrow = mod ? mod + (size_t)(row / rows_per_mod) * 3 * H : nullptr;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    float o[8];
    if (mrow) {
      float sc[8], sh[8];
      load8_at(mrow + i, whole, sc);
      load8_at(mrow + H + i, whole, sh);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = srow[i + j] * rstd * (1.f + sc[j]) + sh[j];
    } else {
      float wf[8];
      if (w) {
        load8_at(w + i, whole, wf);
      } else {   // no weight: plain x * rstd in either form
#pragma unroll
        for (int j = 0; j < 8; ++j) wf[j] = (mode & 1) ? 0.f : 1.f;
      }
      if (mode & 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = srow[i + j] * rstd * (1.f + wf[j]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          o[j] = wf[j] * Num<T>::to_f(Num<T>::from_f(srow[i + j] * rstd));
      }
    }
    store8(y + (size_t)row * ldy + i, o);
  }
}

// The same for rows of at most 8192 values, eight to a thread that holds them: everything a row needs, its weights too, is asked for at once and the
// sum takes one barrier.  A row is one chain of trips to memory, and the kernel above has
// two of them, four barriers and eight-way bank conflicts in it.  Behind a GEMM, fp16, us, that one / this: 50 x 1024
// 2.4 / 2.05, 12 x 4096 3.7 / 2.3.  The kernel above takes longer rows, and operands off their 16-byte boundary.
template <typename T>
__global__ void __launch_bounds__(1024)
rmsnorm_row_kernel(const T* __restrict__ x, const T* __restrict__ residual, const T* __restrict__ w, T* __restrict__ y, T* __restrict__ residual_out,
                   const T* __restrict__ mod, int rows_per_mod, int H, int64_t ldx, int64_t ldy, float eps, int mode) {
  pdl_launch_dependents();
  __shared__ float red[32];
  const int row = blockIdx.x, i = threadIdx.x * 8, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const bool in = i < H, weighted = w && !mod;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  pdl_wait();                                     // the weights may be the previous kernel's as well
  const uint4 wq = weighted && in ? *reinterpret_cast<const uint4*>(w + i) : zero;
  const T* mrow = mod ? mod + (size_t)(row / rows_per_mod) * 3 * H : nullptr;
  const uint4 xq = in ? *reinterpret_cast<const uint4*>(x + (size_t)row * ldx + i) : zero;
  const uint4 rq = residual && in ? *reinterpret_cast<const uint4*>(residual + (size_t)row * ldx + i) : zero;
  const uint4 scq = mrow && in ? *reinterpret_cast<const uint4*>(mrow + i) : zero, shq = mrow && in ? *reinterpret_cast<const uint4*>(mrow + H + i) : zero;
  float f[8], ss = 0.f;
  unpack8<T>(xq, f);
  if (residual) {
    float r[8];
    unpack8<T>(rq, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = Num<T>::to_f(Num<T>::from_f(f[j] + r[j]));
    if (residual_out && in) store8(residual_out + (size_t)row * ldx + i, f);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  const float rstd = rsqrtf(warp_sum(lane < nw ? red[lane] : 0.f) / (float)H + eps);
  if (!in) return;
  float o[8];
  if (mrow) {
    float sc[8], sh[8];
    unpack8<T>(scq, sc);
    unpack8<T>(shq, sh);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = f[j] * rstd * (1.f + sc[j]) + sh[j];
  } else {
    float wf[8];
    unpack8<T>(wq, wf);
    if (!w) {                                     // no weight: plain x * rstd in either form
#pragma unroll
      for (int j = 0; j < 8; ++j) wf[j] = (mode & 1) ? 0.f : 1.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = (mode & 1) ? f[j] * rstd * (1.f + wf[j]) : wf[j] * Num<T>::to_f(Num<T>::from_f(f[j] * rstd));
  }
  store8(y + (size_t)row * ldy + i, o);
}

template <typename T>
__global__ void layernorm_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                 const T* __restrict__ b, T* __restrict__ y, int H, int64_t ldx,
                                 int64_t ldy, float eps, int whole) {
  pdl_prologue();
  extern __shared__ float srow[];
  float* red = srow + H;
  const int row = blockIdx.x;
  const T* xr = x + (size_t)row * ldx;
  float s = 0.f;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    float f[8];
    load8_at(xr + i, whole, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      srow[i + j] = f[j];
      s += f[j];
    }
  }
  const float mean = block_sum(s, red) / (float)H;
  float v = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    const float d = srow[i] - mean;
    v += d * d;
  }
  const float var = block_sum(v, red) / (float)H;
  const float rstd = rsqrtf(var + eps);
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    float wf[8], bf[8], o[8];
    load8_at(w + i, whole, wf);
    if (b) load8_at(b + i, whole, bf);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = (srow[i + j] - mean) * rstd * wf[j] + (b ? bf[j] : 0.f);
    store8(y + (size_t)row * ldy + i, o);
  }
}

// Many rows: a warp per row that holds it in registers, 16-byte pieces 256 values apart, all of them on their way at once; nothing but shuffles
// between the two passes.  A block per row has a barrier in its chain (LayerNorm's four), which it hides as long as an SM has few rows: layernorm_by_warp and
// rmsnorm_by_warp have the lines.  us, block / warp: LayerNorm 3072 x 1152 9.0 / 4.4, 6000 x 2048 25.3 / 15.5; RMSNorm 6000 x 4096 37 / 23.
template <typename T, int NC>
__global__ void __launch_bounds__(128)
rmsnorm_warp_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, const T* __restrict__ mod, int rows_per_mod, int rows, int H,
                    int64_t ldx, int64_t ldy, float eps, int mode) {
  pdl_prologue();
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* xr = x + (size_t)row * ldx;
  uint4 v[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int i = c * 256 + lane * 8;
    v[c] = i < H ? *reinterpret_cast<const uint4*>(xr + i) : make_uint4(0u, 0u, 0u, 0u);
  }
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    float f[8];
    unpack8<T>(v[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  const float rstd = rsqrtf(warp_sum(ss) / (float)H + eps);
  const T* mrow = mod ? mod + (size_t)(row / rows_per_mod) * 3 * H : nullptr;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int i = c * 256 + lane * 8;
    if (i >= H) continue;
    float f[8], o[8];
    unpack8<T>(v[c], f);
    if (mrow) {
      float sc[8], sh[8];
      load8(mrow + i, sc);
      load8(mrow + H + i, sh);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = f[j] * rstd * (1.f + sc[j]) + sh[j];
    } else {
      float wf[8];
      if (w) {
        load8(w + i, wf);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) wf[j] = (mode & 1) ? 0.f : 1.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (mode & 1) ? f[j] * rstd * (1.f + wf[j]) : wf[j] * Num<T>::to_f(Num<T>::from_f(f[j] * rstd));
    }
    store8(y + (size_t)row * ldy + i, o);
  }
}

// Short rows' weights and biases are asked for beside the row (behind its two sums, they were another trip to memory; behind a GEMM, us: 3072 x 1152
// 7.6, so 5.3; 768 x 1152 6.1 / 3.1).
template <typename T, int NC>
__global__ void __launch_bounds__(128)
layernorm_warp_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ b, T* __restrict__ y, int rows, int H, int64_t ldx,
                      int64_t ldy, float eps) {
  constexpr int kEarly = NC <= 5 ? NC : 0;
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 we[kEarly ? kEarly : 1], be[kEarly ? kEarly : 1];
#pragma unroll
  for (int c = 0; c < kEarly; ++c) {
    const int i = c * 256 + lane * 8;
    we[c] = i < H ? *reinterpret_cast<const uint4*>(w + i) : zero;
    be[c] = b && i < H ? *reinterpret_cast<const uint4*>(b + i) : zero;
  }
  if (row >= rows) return;
  const T* xr = x + (size_t)row * ldx;
  uint4 v[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int i = c * 256 + lane * 8;
    v[c] = i < H ? *reinterpret_cast<const uint4*>(xr + i) : zero;
  }
  float s = 0.f, q = 0.f;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    float f[8];
    unpack8<T>(v[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += f[j];
  }
  const float mean = warp_sum(s) / (float)H;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (c * 256 + lane * 8 >= H) continue;
    float f[8];
    unpack8<T>(v[c], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) q += (f[j] - mean) * (f[j] - mean);
  }
  const float rstd = rsqrtf(warp_sum(q) / (float)H + eps);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int i = c * 256 + lane * 8;
    if (i >= H) continue;
    float f[8], wf[8], bf[8], o[8];
    unpack8<T>(v[c], f);
    if (c < kEarly) {
      unpack8<T>(we[c < kEarly ? c : 0], wf);
      unpack8<T>(be[c < kEarly ? c : 0], bf);
    } else {
      load8(w + i, wf);
      if (b) load8(b + i, bf);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = (f[j] - mean) * rstd * wf[j] + (b ? bf[j] : 0.f);
    store8(y + (size_t)row * ldy + i, o);
  }
}

// 256-value pieces of a row that the warp kernels hold
static int warp_pieces(int H) {
  const int nc = ceil_div(H, 256);
  return nc <= 4 ? 4 : nc <= 5 ? 5 : nc <= 8 ? 8 : nc <= 12 ? 12 : 16;
}
// A warp takes its row alone, so it needs several rows per SM to hide its chain, and more of them the longer the row.  LayerNorm, whose block form
// meets at four barriers, fp16, us, block / warp: 296 x 1024 2.6 / 2.9, 400 x 1152 3.6 / 3.3, 768 x 1152 5.6 / 4.0, 768 x 2048 5.9 / 6.2, 1500 x 4096
// 13.2 / 9.1.
static bool layernorm_by_warp(int rows, int H) { return H <= 4096 && 2 * rows >= (H <= 1152 ? 5 : H <= 1536 ? 10 : 20) * sm_count(); }
// RMSNorm's block form has one barrier, and is overtaken where an SM has some 20 thousand values (34 of rows above 1536 values), later with a modulation's two rows.  fp16, us, block / warp: 3072 x 1024 5.2 / 5.6, 4770 x 1024 7.0 / 6.5, 2200 x
// 2048 6.7 / 7.6, 3072 x 2048 8.6 / 8.1, 1100 x 4096 8.4 / 9.8, 1500 x 4096 10.9 / 10.1; modulated 3072 x 1152 6.6 / 7.4, 4770 x 1152 8.8 / 8.0, 3072 x
// 2048 9.4 / 10.1, 3072 x 2560 11.8 / 10.8.  With a residual never: 768 x 1152 3.1 / 6.0, 3072 x 2048 11.2 / 14.0, 9000 x 1536 22.3 / 22.4.
static bool rmsnorm_by_warp(int rows, int H, bool mod, bool residual) {
  const long per_sm = mod ? (H <= 1536 ? 24300 : 48600) : H <= 1536 ? 21600 : 34000;
  return !residual && H <= 4096 && (long)rows * H >= per_sm * sm_count();
}
// Rows of 16-byte pieces: every operand on its boundary (the kernels that go through shared memory take 4-byte ones)
template <typename... P>
static bool whole_pieces(P... p) { return (((reinterpret_cast<uintptr_t>(p) % 16) == 0) && ...); }
template <typename... P>
static bool whole_words(P... p) { return (((reinterpret_cast<uintptr_t>(p) % 4) == 0) && ...); }

// Calls `run` with the piece count and the element type as types.
template <typename Run>
static cudaError_t with_pieces(int nc, int dtype, Run run) {
  auto typed = [&](auto zero) -> cudaError_t {
    switch (nc) {
      case 4: return run(std::integral_constant<int, 4>{}, zero);
      case 5: return run(std::integral_constant<int, 5>{}, zero);
      case 8: return run(std::integral_constant<int, 8>{}, zero);
      case 12: return run(std::integral_constant<int, 12>{}, zero);
      default: return run(std::integral_constant<int, 16>{}, zero);
    }
  };
  return dtype == 0 ? typed(__half{}) : typed(__nv_bfloat16{});
}

template <typename T>
__global__ void l2norm_kernel(const T* __restrict__ x, T* __restrict__ y, int rows, int H,
                              float eps, float out_scale) {
  pdl_prologue();
  // one warp per row
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int l = threadIdx.x & 31;
  const T* xr = x + (size_t)row * H;
  float ss = 0.f;
  for (int i = l; i < H; i += 32) {
    const float f = Num<T>::to_f(xr[i]);
    ss += f * f;
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss + eps) * out_scale;
  for (int i = l; i < H; i += 32) y[(size_t)row * H + i] = Num<T>::from_f(Num<T>::to_f(xr[i]) * r);
}

// x += gate * y  (adaRMS gated residual; gate per token-group [.., 3H] third block)
template <typename T>
__global__ void gated_residual_kernel(T* __restrict__ x, const T* __restrict__ y,
                                      const T* __restrict__ mod, int rows_per_mod, int H,
                                      int64_t total) {
  pdl_prologue();
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= total) return;
  const int row = (int)(i / H), col = (int)(i % H);
  float a[8], b[8], g[8];
  load8(x + i, a);
  load8(y + i, b);
  load8(mod + (size_t)(row / rows_per_mod) * 3 * H + 2 * H + col, g);
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] += g[j] * b[j];
  store8(x + i, a);
}

}  // namespace rf

using namespace rf;

extern "C" int rf_rmsnorm(const void* x, const void* residual, const void* w, void* y,
                          void* residual_out, const void* mod, int rows_per_mod, int rows, int H,
                          int64_t ldx, int64_t ldy, float eps, int mode, int dtype,
                          rf_stream_t stream) {
  RF_SKIP_IF_REPLAYING();
  RF_REQUIRE(rows >= 0 && H > 0 && H % 8 == 0, "rmsnorm H=%d must be a multiple of 8", H);
  RF_REQUIRE(ldx % 8 == 0 && ldy % 8 == 0, "rmsnorm pitches must be multiples of 8");
  RF_REQUIRE(whole_words(x, residual, w, y, residual_out, mod), "rmsnorm operands must lie on even elements");
  if (rows == 0) return RF_OK;
  const int threads = H >= 2048 ? 256 : 128;
  const size_t smem = (size_t)(H + 32) * sizeof(float);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (rows_per_mod <= 0) rows_per_mod = 1;
  const bool whole = whole_pieces(x, residual, w, y, residual_out, mod);
  if (whole && rmsnorm_by_warp(rows, H, mod != nullptr, residual != nullptr)) {
    auto run = [&](auto kNC, auto zero) -> cudaError_t {
      using T = decltype(zero);
      return ::rf::launch_k(rmsnorm_warp_kernel<T, decltype(kNC)::value>, dim3(ceil_div(rows, 4)), dim3(128), 0, s, 1, (const T*)x, (const T*)w, (T*)y,
                            (const T*)mod, rows_per_mod, rows, H, ldx, ldy, eps, mode);
    };
    RF_CUDA_CHECK(with_pieces(warp_pieces(H), dtype, run));
    ::rf::count_launch();
    return RF_OK;
  }
  if (whole && H <= 8192) {
    auto run = [&](auto zero) -> cudaError_t {
      using T = decltype(zero);
      return ::rf::launch_k(rmsnorm_row_kernel<T>, dim3(rows), dim3(round_up(ceil_div(H, 8), 32)), 0, s, 1, (const T*)x, (const T*)residual, (const T*)w, (T*)y,
                            (T*)residual_out, (const T*)mod, rows_per_mod, H, ldx, ldy, eps, mode);
    };
    RF_CUDA_CHECK(dtype == 0 ? run(__half{}) : run(__nv_bfloat16{}));
    ::rf::count_launch();
    return RF_OK;
  }
  if (dtype == 0)
    RF_CUDA_CHECK(::rf::launch_k(rmsnorm_kernel<__half>, dim3(rows), dim3(threads), smem, s, 1, 
        (const __half*)x, (const __half*)residual, (const __half*)w, (__half*)y,
        (__half*)residual_out, (const __half*)mod, rows_per_mod, H, ldx, ldy, eps, mode, (int)whole));
  else
    RF_CUDA_CHECK(::rf::launch_k(rmsnorm_kernel<__nv_bfloat16>, dim3(rows), dim3(threads), smem, s, 1, 
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)residual, (const __nv_bfloat16*)w,
        (__nv_bfloat16*)y, (__nv_bfloat16*)residual_out, (const __nv_bfloat16*)mod, rows_per_mod,
        H, ldx, ldy, eps, mode, (int)whole));
  RF_CUDA_CHECK(cudaGetLastError());
  ::rf::count_launch();
  return RF_OK;
}

extern "C" int rf_layernorm(const void* x, const void* w, const void* b, void* y, int rows, int H,
                            int64_t ldx, int64_t ldy, float eps, int dtype, rf_stream_t stream) {
  RF_SKIP_IF_REPLAYING();
  RF_REQUIRE(rows >= 0 && H > 0 && H % 8 == 0, "layernorm H=%d must be a multiple of 8", H);
  RF_REQUIRE(ldx % 2 == 0 && ldy % 2 == 0, "layernorm pitches must be even (%lld, %lld)", (long long)ldx, (long long)ldy);
  RF_REQUIRE(whole_words(x, w, b, y), "layernorm operands must lie on even elements");
  if (rows == 0) return RF_OK;
  const int threads = H >= 2048 ? 256 : 128;
  const size_t smem = (size_t)(H + 32) * sizeof(float);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool whole = whole_pieces(x, w, b, y) && ldx % 8 == 0 && ldy % 8 == 0;       // every row on its boundary, not the first alone
  if (whole && layernorm_by_warp(rows, H)) {
    auto run = [&](auto kNC, auto zero) -> cudaError_t {
      using T = decltype(zero);
      return ::rf::launch_k(layernorm_warp_kernel<T, decltype(kNC)::value>, dim3(ceil_div(rows, 4)), dim3(128), 0, s, 1, (const T*)x, (const T*)w, (const T*)b,
                            (T*)y, rows, H, ldx, ldy, eps);
    };
    RF_CUDA_CHECK(with_pieces(warp_pieces(H), dtype, run));
    ::rf::count_launch();
    return RF_OK;
  }
  if (dtype == 0)
    RF_CUDA_CHECK(::rf::launch_k(layernorm_kernel<__half>, dim3(rows), dim3(threads), smem, s, 1, (const __half*)x, (const __half*)w,
                                                        (const __half*)b, (__half*)y, H, ldx, ldy,
                                                        eps, (int)whole));
  else
    RF_CUDA_CHECK(::rf::launch_k(layernorm_kernel<__nv_bfloat16>, dim3(rows), dim3(threads), smem, s, 1, 
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b,
        (__nv_bfloat16*)y, H, ldx, ldy, eps, (int)whole));
  RF_CUDA_CHECK(cudaGetLastError());
  ::rf::count_launch();
  return RF_OK;
}

extern "C" int rf_l2norm(const void* x, void* y, int rows, int H, float eps, float out_scale,
                         int dtype, rf_stream_t stream) {
  RF_SKIP_IF_REPLAYING();
  RF_REQUIRE(rows >= 0 && H > 0, "l2norm shape");
  if (rows == 0) return RF_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int wpb = 4;
  const int blocks = ceil_div(rows, wpb);
  if (dtype == 0)
    RF_CUDA_CHECK(::rf::launch_k(l2norm_kernel<__half>, dim3(blocks), dim3(wpb * 32), 0, s, 1, (const __half*)x, (__half*)y, rows, H, eps, out_scale));
  else
    RF_CUDA_CHECK(::rf::launch_k(l2norm_kernel<__nv_bfloat16>, dim3(blocks), dim3(wpb * 32), 0, s, 1, (const __nv_bfloat16*)x,
                                                             (__nv_bfloat16*)y, rows, H, eps, out_scale));
  RF_CUDA_CHECK(cudaGetLastError());
  ::rf::count_launch();
  return RF_OK;
}

extern "C" int rf_gated_residual(void* x, const void* y, const void* mod, int rows_per_mod,
                                 int rows, int H, int dtype, rf_stream_t stream) {
  RF_SKIP_IF_REPLAYING();
  RF_REQUIRE(H % 8 == 0 && rows >= 0, "gated_residual H=%d must be a multiple of 8", H);
  if (rows == 0) return RF_OK;
  const int64_t total = (int64_t)rows * H;
  const int threads = 256;
  const int blocks = (int)((total / 8 + threads - 1) / threads);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (rows_per_mod <= 0) rows_per_mod = 1;
  if (dtype == 0)
    RF_CUDA_CHECK(::rf::launch_k(gated_residual_kernel<__half>, dim3(blocks), dim3(threads), 0, s, 1, (__half*)x, (const __half*)y,
                                                           (const __half*)mod, rows_per_mod, H, total));
  else
    RF_CUDA_CHECK(::rf::launch_k(gated_residual_kernel<__nv_bfloat16>, dim3(blocks), dim3(threads), 0, s, 1, 
        (__nv_bfloat16*)x, (const __nv_bfloat16*)y, (const __nv_bfloat16*)mod, rows_per_mod, H, total));
  RF_CUDA_CHECK(cudaGetLastError());
  ::rf::count_launch();
  return RF_OK;
}
