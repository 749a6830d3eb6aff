// HBM-bound kernels of the Llama training step: embedding, RMSNorm (+ residual add),
// RoPE, SwiGLU, fused softmax cross-entropy, fused AdamW, gradient-norm.  All tensors
// are bf16 unless stated, rows are contiguous, and every row length must be a multiple
// of 8 elements so that all traffic is 16-byte vectors.
#include <algorithm>
#include <type_traits>

#include "ftb200_common.cuh"
#include "tcgen05_helpers.cuh"

using ftb200::bf16x8;
using ftb200::pack8;
using ftb200::unpack8;

namespace {

// ------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const int64_t* tok, const bf16x8* table,
                                     bf16x8* out, int T, int D8, int V) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int t = blockIdx.x;
  if (t >= T) return;
  int64_t id = tok[t];
  if (!FTB_IN_RANGE(id, V) || id < 0 || id >= V) id = 0;  // an id outside the vocabulary reads row 0
  const bf16x8* src = table + id * D8;
  bf16x8* dst = out + static_cast<int64_t>(t) * D8;
  for (int i = threadIdx.x; i < D8; i += blockDim.x) dst[i] = src[i];
}

__global__ void embedding_bwd_kernel(const int64_t* tok, const __nv_bfloat162* dout,
                                     __nv_bfloat162* dtable, int T, int D2, int V) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int t = blockIdx.x;
  if (t >= T) return;
  int64_t id = tok[t];
  if (!FTB_IN_RANGE(id, V) || id < 0 || id >= V) return;
  const __nv_bfloat162* src = dout + static_cast<int64_t>(t) * D2;
  __nv_bfloat162* dst = dtable + id * D2;
  for (int i = threadIdx.x; i < D2; i += blockDim.x) atomicAdd(dst + i, src[i]);
}

// ------------------------------------------------------------------ RMSNorm
// Rows are worked on by groups of TPR threads (one to eight warps), each thread with VPT vectors of 8 elements that stay in
// registers, packed, between the reduction and the second use.
template <int TPR>
__device__ __forceinline__ float group_sum(float v, float* part) {
  v = ftb200::warp_sum(v);
  if constexpr (TPR > 32) {
    // one barrier of the group's own: callers that come here again alternate between two sets of `part`
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    const int g = threadIdx.x / TPR;
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(TPR) : "memory");
    v = 0.f;
#pragma unroll
    for (int k = 0; k < TPR / 32; ++k) v += part[g * (TPR / 32) + k];
  }
  return v;
}

constexpr int NORM_THREADS = 256;

// out = x * rstd * w ;  optionally first h = x + res (written to h_out) and normalise h.  Bound by memory (by L2 where the
// rows fit there): every vector is read once, all of a thread's loads are in flight together, and the 256 / TPR rows of
// a block wait for nothing of each other's.  With a block per row, read twice around three barriers: 63.3 us for
// 8192 x 4096 (51.8 now, 5.2 TB/s), 32.4 for 8192 x 2048 (28.0), 9.5 for 3000 x 1024 (7.8).
template <int TPR, int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const bf16x8* x, const bf16x8* res, bf16x8* h_out,
                   const bf16x8* w, bf16x8* out, float* rstd_out, int T, int D8,
                   float eps) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  __shared__ float part[NORM_THREADS / 32];
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (NORM_THREADS / TPR) + threadIdx.x / TPR;
  if (row >= T) return;  // a whole group
  const int i0 = threadIdx.x % TPR;
  bf16x8 a[VPT], c[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = i0 + v * TPR;
    if (i < D8) {
      a[v] = x[row * D8 + i];
      if (res != nullptr) c[v] = res[row * D8 + i];
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = i0 + v * TPR;
    if (i < D8) {
      float f[8];
      unpack8(a[v], f);
      if (res != nullptr) {
        float g[8];
        unpack8(c[v], g);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += g[e];
        a[v] = pack8(f);
        h_out[row * D8 + i] = a[v];
        unpack8(a[v], f);  // normalise the rounded value that later passes will read
      }
      c[v] = w[i];  // on its way during the reduction
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
    }
  }
  ss = group_sum<TPR>(ss, part);
  const float r = rsqrtf(ss / (8.f * D8) + eps);
  if (i0 == 0 && rstd_out != nullptr) rstd_out[row] = r;
  if (out == nullptr) return;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = i0 + v * TPR;
    if (i < D8) {
      float f[8], g[8];
      unpack8(a[v], f);
      unpack8(c[v], g);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = f[e] * r * g[e];
      out[row * D8 + i] = pack8(f);
    }
  }
}

// The same for rows longer than 8192 elements: a block per row, which is read twice.
__global__ void rmsnorm_fwd_long_kernel(const bf16x8* x, const bf16x8* res,
                                        bf16x8* h_out, const bf16x8* w,
                                        bf16x8* out, float* rstd_out, int D8, float eps) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  __shared__ float scratch[33];
  const int64_t row = blockIdx.x;
  const bf16x8* xr = x + row * D8;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D8; i += blockDim.x) {
    float f[8];
    unpack8(xr[i], f);
    if (res != nullptr) {
      float g[8];
      unpack8(res[row * D8 + i], g);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] += g[e];
      bf16x8 hv = pack8(f);
      h_out[row * D8 + i] = hv;
      unpack8(hv, f);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
  }
  ss = ftb200::block_sum(ss, scratch);
  const float r = rsqrtf(ss / (8.f * D8) + eps);
  if (threadIdx.x == 0 && rstd_out != nullptr) rstd_out[row] = r;
  if (out == nullptr) return;
  const bf16x8* src = (res != nullptr) ? (h_out + row * D8) : xr;
  for (int i = threadIdx.x; i < D8; i += blockDim.x) {
    float f[8], g[8];
    unpack8(src[i], f);
    unpack8(w[i], g);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = f[e] * r * g[e];
    out[row * D8 + i] = pack8(f);
  }
}

constexpr int NORM_BWD_THREADS = 512;

// dx = dres + rstd*w*dy - x*rstd^3/D * sum(dy*w*x);  dw partial sums per block.
// A group keeps its columns over all its rows, so dw accumulates in registers; the groups of a block meet in shared memory
// at the end and leave one row of partial sums.  One block per SM, 2 to 16 groups in it: what a row waits for (its loads,
// its reduction) is covered by the rows of the other groups, which nothing ties to it.  Two rows a block and iteration around one block-wide sum, two blocks per SM, 296 rows of partial sums:
// 8192 x 2048 45.3 us (38.0 now, both kernels), 3000 x 1024 19.4 (14.0), 2500 x 8192 60.9 (50.7), 8192 x 4096 67.8 (66.8).
template <int TPR, int VPT>
__global__ void __launch_bounds__(NORM_BWD_THREADS, 1)
rmsnorm_bwd_kernel(const bf16x8* dy, const bf16x8* x, const bf16x8* w,
                   const float* rstd, const bf16x8* dres, bf16x8* dx,
                   float* dw_partial, int T, int D8) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  constexpr int GROUPS = NORM_BWD_THREADS / TPR;
  __shared__ float part[2][NORM_BWD_THREADS / 32];
  __shared__ float4 dw_groups[NORM_BWD_THREADS][2];
  const int g = threadIdx.x / TPR, i0 = threadIdx.x % TPR;
  float dw_acc[VPT][8];
#pragma unroll
  for (int v = 0; v < VPT; ++v)
#pragma unroll
    for (int e = 0; e < 8; ++e) dw_acc[v][e] = 0.f;
  int turn = 0;
  for (int64_t row = blockIdx.x + static_cast<int64_t>(gridDim.x) * g; row < T; row += static_cast<int64_t>(gridDim.x) * GROUPS) {
    bf16x8 a[VPT], b[VPT], d[VPT];
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int i = i0 + v * TPR;
      if (i < D8) {
        a[v] = dy[row * D8 + i];
        b[v] = x[row * D8 + i];
        if (dres != nullptr) d[v] = dres[row * D8 + i];
      }
    }
    const float r = rstd[row];
    float dot = 0.f;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      if (i0 + v * TPR < D8) {
        float fa[8], fb[8], c[8];
        unpack8(a[v], fa);
        unpack8(b[v], fb);
        unpack8(w[i0 + v * TPR], c);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          dot += fa[e] * c[e] * fb[e];
          dw_acc[v][e] += fa[e] * fb[e] * r;
        }
      }
    }
    dot = group_sum<TPR>(dot, part[turn]);
    turn ^= 1;
    const float coef = dot * r * r * r / (8.f * D8);
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int i = i0 + v * TPR;
      if (i < D8) {
        float fa[8], fb[8], c[8], o[8];
        unpack8(a[v], fa);
        unpack8(b[v], fb);
        unpack8(w[i0 + v * TPR], c);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = r * c[e] * fa[e] - fb[e] * coef;
        if (dres != nullptr) {
          float fd[8];
          unpack8(d[v], fd);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += fd[e];
        }
        dx[row * D8 + i] = pack8(o);
      }
    }
  }
  float4* dst = reinterpret_cast<float4*>(dw_partial) + static_cast<int64_t>(blockIdx.x) * (2 * D8);
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    if (v > 0) __syncthreads();
    dw_groups[threadIdx.x][0] = make_float4(dw_acc[v][0], dw_acc[v][1], dw_acc[v][2], dw_acc[v][3]);
    dw_groups[threadIdx.x][1] = make_float4(dw_acc[v][4], dw_acc[v][5], dw_acc[v][6], dw_acc[v][7]);
    __syncthreads();
    const int c = threadIdx.x;  // four columns of the group's 8 TPR
    if (c < 2 * TPR && v * 2 * TPR + c < 2 * D8) {
      float4 s = dw_groups[c >> 1][c & 1];
#pragma unroll
      for (int k = 1; k < GROUPS; ++k) {
        const float4 t = dw_groups[k * TPR + (c >> 1)][c & 1];
        s.x += t.x;
        s.y += t.y;
        s.z += t.z;
        s.w += t.w;
      }
      dst[v * 2 * TPR + c] = s;
    }
  }
}

// dw[c] (+)= sum_b partial[b][c].  A block owns 32 columns; its 32 warps stride over the rows (each warp instruction reads
// one 128-byte row segment) and meet in shared memory: a row of partial sums per SM is five independent loads a thread.
__global__ void __launch_bounds__(1024) colsum_partials_kernel(const float* partial, __nv_bfloat16* dw,
                                                               int nblk, int D, int accumulate) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  __shared__ float red[32][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < D) {
#pragma unroll 5
    for (int b = ry; b < nblk; b += 32) s += partial[static_cast<int64_t>(b) * D + c];
  }
  red[ry][cx] = s;
  __syncthreads();
  const float t = ftb200::warp_sum(red[cx][ry]);  // warp ry: column ry of the block, lane cx: row cx of the sums
  const int col = blockIdx.x * 32 + ry;
  if (cx == 0 && col < D) dw[col] = __float2bfloat16(accumulate ? t + __bfloat162float(dw[col]) : t);
}

// Threads per row and vectors per thread: as few warps a row as 4 vectors a thread allow (8 loads of 16 bytes in flight in
// the forward pass, 12 in the backward pass), up to 8 warps for 8192 elements.  With `few` rows, which leave the SMs room,
// twice the threads and half the vectors: 64 x 1024 3.6 -> 2.8 us forward, but 3000 x 1024 7.8 -> 9.3.
template <typename F>
int with_row_shape(int D8, bool few, F&& f) {
  if (few && D8 > 64 && D8 <= 128) return f(std::integral_constant<int, 64>(), std::integral_constant<int, 2>());
  if (few && D8 > 128 && D8 <= 256) return f(std::integral_constant<int, 128>(), std::integral_constant<int, 2>());
  if (few && D8 > 256 && D8 <= 512) return f(std::integral_constant<int, 256>(), std::integral_constant<int, 2>());
  if (D8 <= 32) return f(std::integral_constant<int, 32>(), std::integral_constant<int, 1>());
  if (D8 <= 64) return f(std::integral_constant<int, 32>(), std::integral_constant<int, 2>());
  if (D8 <= 128) return f(std::integral_constant<int, 32>(), std::integral_constant<int, 4>());
  if (D8 <= 256) return f(std::integral_constant<int, 64>(), std::integral_constant<int, 4>());
  if (D8 <= 512) return f(std::integral_constant<int, 128>(), std::integral_constant<int, 4>());
  if (D8 <= 1024) return f(std::integral_constant<int, 256>(), std::integral_constant<int, 4>());
  return FTB200_E_TOOBIG;
}

// Both kernels of the backward pass; dw_partial holds at least min(T, SMs) * D floats.
int launch_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx, void* dw,
                       float* dw_partial, int T, int D, int accumulate_dw, int sms, cudaStream_t st) {
  const int D8 = D / 8;
  return with_row_shape(D8, T <= sms, [&](auto tpr, auto vpt) {
    constexpr int GROUPS = NORM_BWD_THREADS / tpr;
    const int nblk = std::min((T + 3) / 4, sms);
    ftb200::launch_after(rmsnorm_bwd_kernel<tpr, vpt>, nblk, NORM_BWD_THREADS, 0, st, (const bf16x8*)dy, (const bf16x8*)x,
        (const bf16x8*)w, rstd, (const bf16x8*)dres, (bf16x8*)dx, dw_partial, T, D8);
    ftb200::launch_after(colsum_partials_kernel, (D + 31) / 32, 1024, 0, st, dw_partial, (__nv_bfloat16*)dw, nblk, D,
        accumulate_dw);
    return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
  });
}

// ------------------------------------------------------------------ RoPE (interleaved pairs)
// buf rows are [n_rot_heads * Dh | untouched tail]; cs = [S, Dh/2] of (cos, sin).
// One thread rotates 8 consecutive elements (4 pairs): one 16-byte load/store of data and
// two 16-byte loads of the table.
__global__ void rope_kernel(bf16x8* buf, const float4* cs, int64_t T, int S, int n_heads,
                            int Dh8, int64_t row_stride8, float sin_sign) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t per_row = static_cast<int64_t>(n_heads) * Dh8;
  if (idx >= T * per_row) return;
  const int64_t t = idx / per_row;
  const int r = static_cast<int>(idx - t * per_row);
  const int v = r % Dh8;  // which group of 4 pairs inside the head
  const int pos = static_cast<int>(t % S);
  const float4* c = cs + (static_cast<int64_t>(pos) * Dh8 + v) * 2;  // 4 (cos, sin) pairs = 2 float4
  const float4 c0 = c[0], c1 = c[1];
  const float cosv[4] = {c0.x, c0.z, c1.x, c1.z};
  const float sinv[4] = {c0.y * sin_sign, c0.w * sin_sign, c1.y * sin_sign, c1.w * sin_sign};
  if (!FTB_IN_RANGE(r, row_stride8)) return;  // rotated heads must fit inside a row
  bf16x8* p = buf + t * row_stride8 + r;
  float f[8];
  unpack8(*p, f);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float a = f[2 * e], b = f[2 * e + 1];
    f[2 * e] = a * cosv[e] - b * sinv[e];
    f[2 * e + 1] = a * sinv[e] + b * cosv[e];
  }
  *p = pack8(f);
}

// ------------------------------------------------------------------ SwiGLU
// gu rows hold interleaved (gate_j, up_j) pairs: [g0 u0 g1 u1 ...] (2F values);
// out[j] = silu(g_j) * u_j.  One thread handles 4 pairs.
__device__ __forceinline__ void store4_bf16(__nv_bfloat16* p, const float* f) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
  uint2 o;
  o.x = *reinterpret_cast<uint32_t*>(&lo);
  o.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = o;
}

__global__ void swiglu_fwd_kernel(const bf16x8* gu, __nv_bfloat16* out, int64_t n8) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= n8) return;
  float f[8], o[4];
  unpack8(gu[idx], f);
#pragma unroll
  for (int e = 0; e < 4; ++e) o[e] = f[2 * e] / (1.f + __expf(-f[2 * e])) * f[2 * e + 1];
  store4_bf16(out + idx * 4, o);
}

// dgu pair = (ds * u * dsilu(g), ds * silu(g))   (may alias gu: in place)
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* ds, const bf16x8* gu, bf16x8* dgu, int64_t n8) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= n8) return;
  float f[8], o[8];
  unpack8(gu[idx], f);
  const uint2 raw = *reinterpret_cast<const uint2*>(ds + idx * 4);
  const float2 d01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 d23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  const float d[4] = {d01.x, d01.y, d23.x, d23.y};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float g = f[2 * e], u = f[2 * e + 1];
    const float sg = 1.f / (1.f + __expf(-g));
    const float silu = g * sg;
    o[2 * e] = d[e] * u * (sg + silu * (1.f - sg));
    o[2 * e + 1] = d[e] * silu;
  }
  dgu[idx] = pack8(o);
}

// ------------------------------------------------------------------ cross-entropy
// One block per row.  loss[row] = logsumexp(row) - row[target]; with `grad` the row is overwritten in place by
// (softmax - onehot) * grad_scale, without it it is only read.  Bound by memory: a row is read from DRAM and written once, and
// read a second time from the L2, last pieces first (they are the likeliest still there) and, like the writes, without a claim to
// stay.  The exponential unit (two an element) and the issue slots come next, hence packed pairs, no one-hot test outside
// the target's vector, and blocks of 512: three on an SM are seldom all in the same pass, and have the registers for four loads
// in flight.  8192 x 128256 1015 -> 778 us (5.4 TB/s), 4096 x 50304 221 -> 156, 1024 x 32000 45 -> 35, 750 x 8192 18 -> 14;
// in blocks of 1024, two loads, 769, 172, 35, 16; first pieces first 847, 176, 39, 16.
constexpr int CE_LOADS = 4, CE_THREADS = 512;

__global__ void __launch_bounds__(CE_THREADS, 3)
cross_entropy_kernel(bf16x8* logits, const int64_t* target, float* loss, int V8, int64_t ld8, float grad_scale, int grad) {
  using namespace ftb200::tc;
  ftb200::wait_for_previous();
  ftb200::start_next();
  __shared__ float scratch[33];
  const int64_t row = blockIdx.x;
  bf16x8* lr = logits + row * ld8;
  const unsigned long long log2e = f2_pack(1.4426950408889634f, 1.4426950408889634f);
  // exp(x + d) of two
  auto exp_of = [&](float x0, float x1, unsigned long long d) {
    float y0, y1;
    f2_unpack(f2_mul(f2_add(f2_pack(x0, x1), d), log2e), y0, y1);
    return f2_pack(exp2f(y0), exp2f(y1));
  };
  float mx = -INFINITY;
  unsigned long long sum2 = 0ull;
  auto take = [&](const bf16x8& v) {
    float f[8];
    unpack8(v, f);
    float cm = f[0];
#pragma unroll
    for (int e = 1; e < 8; ++e) cm = fmaxf(cm, f[e]);
    if (cm > mx) {
      const float a = __expf(mx - cm);
      sum2 = f2_mul(sum2, f2_pack(a, a));
      mx = cm;
    }
    const unsigned long long neg_mx = f2_pack(-mx, -mx);
#pragma unroll
    for (int e = 0; e < 8; e += 2) sum2 = f2_add(sum2, exp_of(f[e], f[e + 1], neg_mx));
  };
  int i = threadIdx.x;
  for (; i + (CE_LOADS - 1) * CE_THREADS < V8; i += CE_LOADS * CE_THREADS) {
    bf16x8 v[CE_LOADS];
#pragma unroll
    for (int u = 0; u < CE_LOADS; ++u) v[u] = lr[i + u * CE_THREADS];
#pragma unroll
    for (int u = 0; u < CE_LOADS; ++u) take(v[u]);
  }
  for (; i < V8; i += CE_THREADS) take(lr[i]);
  float sum, sum_odd;
  f2_unpack(sum2, sum, sum_odd);
  sum += sum_odd;
  const float gmx = ftb200::block_max(mx, scratch);
  sum *= __expf(mx - gmx);
  const float gsum = ftb200::block_sum(sum, scratch);
  const int64_t tgt = target[row];
  if (tgt >= 0) (void)FTB_IN_RANGE(tgt, 8 * static_cast<int64_t>(V8));  // negative targets mean "ignore"
  (void)FTB_IN_RANGE(V8 - 1, ld8);                                        // a row must fit inside its stride
  const float inv = 1.f / gsum;
  const bool inside = tgt >= 0 && tgt < 8 * static_cast<int64_t>(V8);
  if (threadIdx.x == 0) {
    const __nv_bfloat16* flat = reinterpret_cast<const __nv_bfloat16*>(lr);
    loss[row] = (tgt >= 0) ? (logf(gsum) + gmx - (inside ? __bfloat162float(flat[tgt]) : 0.f)) : 0.f;
  }
  if (!grad) return;
  __syncthreads();  // the target logit is read before any thread overwrites it
  const float gs = (tgt >= 0) ? grad_scale : 0.f;
  const int tgt8 = inside ? static_cast<int>(tgt >> 3) : -1, tgt_e = static_cast<int>(tgt & 7);
  const unsigned long long neg_gmx = f2_pack(-gmx, -gmx), scale2 = f2_pack(inv * gs, inv * gs);
  auto put = [&](const uint4& raw, int at) {
    float f[8];
    unpack8(*reinterpret_cast<const bf16x8*>(&raw), f);
    if (at != tgt8) {
#pragma unroll
      for (int e = 0; e < 8; e += 2) f2_unpack(f2_mul(exp_of(f[e], f[e + 1], neg_gmx), scale2), f[e], f[e + 1]);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = (__expf(f[e] - gmx) * inv - (e == tgt_e ? 1.f : 0.f)) * gs;
    }
    const bf16x8 out = pack8(f);
    __stcs(reinterpret_cast<uint4*>(lr + at), *reinterpret_cast<const uint4*>(&out));
  };
  const uint4* src = reinterpret_cast<const uint4*>(lr);
  if (static_cast<int>(threadIdx.x) >= V8) return;
  i = threadIdx.x + (V8 - 1 - static_cast<int>(threadIdx.x)) / CE_THREADS * CE_THREADS;  // this thread's last
  for (; i - (CE_LOADS - 1) * CE_THREADS >= 0; i -= CE_LOADS * CE_THREADS) {
    uint4 v[CE_LOADS];
#pragma unroll
    for (int u = 0; u < CE_LOADS; ++u) v[u] = __ldcs(src + i - u * CE_THREADS);
#pragma unroll
    for (int u = 0; u < CE_LOADS; ++u) put(v[u], i - u * CE_THREADS);
  }
  for (; i >= 0; i -= CE_THREADS) put(__ldcs(src + i), i);
}

// loss[row] from the maxima, sums and target values that the tiles of a product noted (ftb200_gemm_bf16_loss), a warp a row.
__global__ void __launch_bounds__(256)
cross_entropy_rows_kernel(const long long* target, const float2* stats,
                          const float* target_value, float* loss, int tiles, int T, long long V) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= T) return;
  const float2* st = stats + row * tiles;
  float mx = -INFINITY, sum = 0.f;
  for (int i = lane; i < tiles; i += 32) mx = fmaxf(mx, st[i].x);
  mx = ftb200::warp_max(mx);
  const float base = mx == -INFINITY ? 0.f : mx;
  for (int i = lane; i < tiles; i += 32) sum += st[i].y * __expf(st[i].x - base);
  sum = ftb200::warp_sum(sum);
  const long long tgt = target[row];
  if (lane == 0) {
    if (tgt >= 0) (void)FTB_IN_RANGE(tgt, V);
    loss[row] = tgt >= 0 ? logf(sum) + mx - (tgt < V ? target_value[row] : 0.f) : 0.f;
  }
}

// ------------------------------------------------------------------ AdamW (flat shard)
// master/m/v fp32, grad bf16 or fp32, writes the bf16 working copy.  `grad_scale_dev`
// (optional) is a device scalar multiplied into every gradient (clipping coefficient).
template <typename G>
__global__ void adamw_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                             const G* __restrict__ grad, __nv_bfloat16* __restrict__ param_bf16, int64_t n, float lr,
                             float beta1, float beta2, float eps, float wd, float bc1, float bc2_sqrt,
                             const float* __restrict__ grad_scale_dev) {
  const float gs = grad_scale_dev ? *grad_scale_dev : 1.f;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x * 4;
  for (int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4; i < n; i += stride) {
    if (i + 4 <= n) {
      float4 p4 = *reinterpret_cast<float4*>(master + i);
      float4 m4 = *reinterpret_cast<float4*>(m + i);
      float4 v4 = *reinterpret_cast<float4*>(v + i);
      float g[4];
      if constexpr (sizeof(G) == 2) {
        const uint2 raw = *reinterpret_cast<const uint2*>(grad + i);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        g[0] = a.x; g[1] = a.y; g[2] = b.x; g[3] = b.y;
      } else {
        const float4 gg = *reinterpret_cast<const float4*>(grad + i);
        g[0] = gg.x; g[1] = gg.y; g[2] = gg.z; g[3] = gg.w;
      }
      float* pp = &p4.x;
      float* mm = &m4.x;
      float* vv = &v4.x;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float ge = g[e] * gs;
        mm[e] = beta1 * mm[e] + (1.f - beta1) * ge;
        vv[e] = beta2 * vv[e] + (1.f - beta2) * ge * ge;
        const float denom = sqrtf(vv[e]) / bc2_sqrt + eps;
        pp[e] = pp[e] * (1.f - lr * wd) - (lr / bc1) * (mm[e] / denom);
      }
      *reinterpret_cast<float4*>(master + i) = p4;
      *reinterpret_cast<float4*>(m + i) = m4;
      *reinterpret_cast<float4*>(v + i) = v4;
      if (param_bf16 != nullptr) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(p4.x, p4.y), hi = __floats2bfloat162_rn(p4.z, p4.w);
        uint2 o;
        o.x = *reinterpret_cast<uint32_t*>(&lo);
        o.y = *reinterpret_cast<uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(param_bf16 + i) = o;
      }
    } else {
      for (int64_t j = i; j < n; ++j) {
        float ge;
        if constexpr (sizeof(G) == 2) ge = __bfloat162float(grad[j]) * gs; else ge = grad[j] * gs;
        const float mj = beta1 * m[j] + (1.f - beta1) * ge;
        const float vj = beta2 * v[j] + (1.f - beta2) * ge * ge;
        const float denom = sqrtf(vj) / bc2_sqrt + eps;
        const float pj = master[j] * (1.f - lr * wd) - (lr / bc1) * (mj / denom);
        m[j] = mj; v[j] = vj; master[j] = pj;
        if (param_bf16 != nullptr) param_bf16[j] = __float2bfloat16(pj);
      }
    }
  }
}

// sum of squares of a bf16 (or fp32) buffer, accumulated into *out with one atomic per block.
template <typename G>
__global__ void sumsq_kernel(const G* x, int64_t n, float* out) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  __shared__ float scratch[33];
  float s = 0.f;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  if constexpr (sizeof(G) == 2) {
    const int64_t n8 = n / 8;
    const bf16x8* xv = reinterpret_cast<const bf16x8*>(x);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8; i += stride) {
      float f[8];
      unpack8(xv[i], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) s += f[e] * f[e];
    }
    for (int64_t j = n8 * 8 + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += stride) {
      const float f = __bfloat162float(x[j]);
      s += f * f;
    }
  } else {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) s += x[i] * x[i];
  }
  s = ftb200::block_sum(s, scratch);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// coef = min(1, max_norm / (sqrt(sumsq) + 1e-6)); also stores the norm.
__global__ void clip_coef_kernel(const float* sumsq, float max_norm, float* coef,
                                 float* norm_out) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const float nrm = sqrtf(*sumsq);
  if (norm_out) *norm_out = nrm;
  *coef = (max_norm > 0.f) ? fminf(1.f, max_norm / (nrm + 1e-6f)) : 1.f;
}

int grid_for(int64_t work_items, int block) {
  int64_t g = (work_items + block - 1) / block;
  return static_cast<int>(g < 1 ? 1 : g);
}

}  // namespace

FTB200_API int ftb200_embedding_fwd(const int64_t* tok, const void* table, void* out, int T, int D, int V,
                                    cudaStream_t st) {
  if (D % 8) return FTB200_E_ALIGN;
  ftb200::launch_after(embedding_fwd_kernel, T, 256, 0, st, tok, (const bf16x8*)table, (bf16x8*)out, T, D / 8, V);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

FTB200_API int ftb200_embedding_bwd(const int64_t* tok, const void* dout, void* dtable, int T, int D, int V,
                                    cudaStream_t st) {
  if (D % 8) return FTB200_E_ALIGN;
  ftb200::launch_after(embedding_bwd_kernel, T, 256, 0, st, tok, (const __nv_bfloat162*)dout, (__nv_bfloat162*)dtable, T,
      D / 2, V);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

// res/h_out may be null (plain norm); out may be null (only rstd wanted).
FTB200_API int ftb200_rmsnorm_fwd(const void* x, const void* res, void* h_out, const void* w, void* out, float* rstd,
                                  int T, int D, float eps, cudaStream_t st) {
  if (D % 8) return FTB200_E_ALIGN;
  if (res != nullptr && h_out == nullptr) return FTB200_E_BADARG;
  const int D8 = D / 8;
  const int rc = with_row_shape(D8, T <= 4 * ftb200::sm_count(), [&](auto tpr, auto vpt) {
    constexpr int ROWS = NORM_THREADS / tpr;
    ftb200::launch_after(rmsnorm_fwd_kernel<tpr, vpt>, (T + ROWS - 1) / ROWS, NORM_THREADS, 0, st, (const bf16x8*)x,
        (const bf16x8*)res, (bf16x8*)h_out, (const bf16x8*)w, (bf16x8*)out, rstd, T, D8, eps);
    return 0;
  });
  if (rc != 0)
    ftb200::launch_after(rmsnorm_fwd_long_kernel, T, 512, 0, st, (const bf16x8*)x, (const bf16x8*)res, (bf16x8*)h_out,
        (const bf16x8*)w, (bf16x8*)out, rstd, D8, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

// Number of floats the caller must provide in `dw_partial` for ftb200_rmsnorm_bwd.
FTB200_API long long ftb200_rmsnorm_bwd_scratch_floats(int D) {
  return static_cast<long long>(ftb200::sm_count()) * 2 * D;
}

FTB200_API int ftb200_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                                  void* dx, void* dw, float* dw_partial, int T, int D, int accumulate_dw,
                                  cudaStream_t st) {
  if (D % 8) return FTB200_E_ALIGN;
  return launch_rmsnorm_bwd(dy, x, w, rstd, dres, dx, dw, dw_partial, T, D, accumulate_dw, ftb200::sm_count(), st);
}

// Rotates the first n_heads heads of every row in place.  backward != 0 applies the inverse rotation.
FTB200_API int ftb200_rope(void* buf, const float* cos_sin, long long T, int S, int n_heads, int head_dim,
                           long long row_stride, int backward, cudaStream_t st) {
  if (head_dim % 8 || row_stride % 8 || (reinterpret_cast<uintptr_t>(buf) & 15)) return FTB200_E_ALIGN;
  const int64_t total = T * n_heads * (head_dim / 8);
  ftb200::launch_after(rope_kernel, grid_for(total, 256), 256, 0, st, (bf16x8*)buf, (const float4*)cos_sin, T, S, n_heads,
      head_dim / 8, row_stride / 8, backward ? -1.f : 1.f);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

FTB200_API int ftb200_swiglu_fwd(const void* gu, void* out, long long T, int F, cudaStream_t st) {
  if (F % 4) return FTB200_E_ALIGN;
  const int64_t n8 = T * (F / 4);
  ftb200::launch_after(swiglu_fwd_kernel, grid_for(n8, 256), 256, 0, st, (const bf16x8*)gu, (__nv_bfloat16*)out, n8);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

FTB200_API int ftb200_swiglu_bwd(const void* ds, const void* gu, void* dgu, long long T, int F, cudaStream_t st) {
  if (F % 4) return FTB200_E_ALIGN;
  const int64_t n8 = T * (F / 4);
  ftb200::launch_after(swiglu_bwd_kernel, grid_for(n8, 256), 256, 0, st, (const __nv_bfloat16*)ds, (const bf16x8*)gu,
      (bf16x8*)dgu, n8);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

FTB200_API int ftb200_cross_entropy(void* logits, const int64_t* target, float* loss, int T, int V, long long ld,
                                    float grad_scale, int grad, cudaStream_t st) {
  if (V % 8 || ld % 8) return FTB200_E_ALIGN;
  ftb200::launch_after(cross_entropy_kernel, T, CE_THREADS, 0, st, (bf16x8*)logits, target, loss, V / 8, ld / 8, grad_scale, grad);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

// Second half of ftb200_gemm_bf16_loss.
int ftb200_launch_cross_entropy_rows(const long long* target, const float2* row_stats, const float* target_value, float* loss,
                                     int tiles, int T, int V, cudaStream_t st) {
  ftb200::launch_after(cross_entropy_rows_kernel, (T + 7) / 8, 256, 0, st, target, row_stats, target_value, loss, tiles, T, V);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

FTB200_API int ftb200_adamw(float* master, float* m, float* v, const void* grad, int grad_is_fp32, void* param_bf16,
                            long long n, float lr, float beta1, float beta2, float eps, float wd, int step,
                            const float* grad_scale_dev, cudaStream_t st) {
  if (n <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15)
    return FTB200_E_ALIGN;
  if (reinterpret_cast<uintptr_t>(grad) & (grad_is_fp32 ? 15 : 7)) return FTB200_E_ALIGN;
  if (reinterpret_cast<uintptr_t>(param_bf16) & 7) return FTB200_E_ALIGN;
  const float bc1 = 1.f - powf(beta1, static_cast<float>(step));
  const float bc2s = sqrtf(1.f - powf(beta2, static_cast<float>(step)));
  // One pass of the loop per thread: blocks that come and go keep reads and writes apart less than 16 long-lived ones per
  // SM in step do.  1.9 G parameters 8869 -> 7777 us (6840 GB/s).
  const int blocks = static_cast<int>(std::min<long long>((n / 4 + 255) / 256 + 1, 0x7fffffffLL));
  if (grad_is_fp32)
    adamw_kernel<float><<<blocks, 256, 0, st>>>(master, m, v, (const float*)grad, (__nv_bfloat16*)param_bf16, n, lr,
                                                beta1, beta2, eps, wd, bc1, bc2s, grad_scale_dev);
  else
    adamw_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(master, m, v, (const __nv_bfloat16*)grad,
                                                        (__nv_bfloat16*)param_bf16, n, lr, beta1, beta2, eps, wd, bc1,
                                                        bc2s, grad_scale_dev);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

// *out += sum(x^2).  The caller zeroes *out before the first call of a step.
FTB200_API int ftb200_sumsq(const void* x, int is_fp32, long long n, float* out, cudaStream_t st) {
  if (n <= 0) return 0;
  if (reinterpret_cast<uintptr_t>(x) & 15) return FTB200_E_ALIGN;
  const int blocks = static_cast<int>(std::min<long long>((n / 8 + 255) / 256 + 1, ftb200::sm_count() * 8LL));
  if (is_fp32)
    ftb200::launch_after(sumsq_kernel<float>, blocks, 256, 0, st, (const float*)x, n, out);
  else
    ftb200::launch_after(sumsq_kernel<__nv_bfloat16>, blocks, 256, 0, st, (const __nv_bfloat16*)x, n, out);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

FTB200_API int ftb200_clip_coef(const float* sumsq, float max_norm, float* coef, float* norm_out, cudaStream_t st) {
  ftb200::launch_after(clip_coef_kernel, 1, 1, 0, st, sumsq, max_norm, coef, norm_out);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

// ------------------------------------------------------------------ allocation-free variant
// See ftb200_noalloc.h.  The scratch lives in the library image; host code must not pass
// the symbol itself to a kernel (on the host it is only a stand-in), so its device address
// is looked up once per device and cached.
#include <atomic>

#include "ftb200_noalloc.h"

static __device__ __align__(256) float g_noalloc_scratch[FTB200_NOALLOC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
// Host threads may make their first call on a device at the same time: they all resolve the
// same address, and the atomic makes the concurrent store and loads well defined.
std::atomic<float*> g_noalloc_scratch_addr[kMaxDevices];
}  // namespace

FTB200_API int ftb200_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd,
                                          const void* dres, void* dx, void* dw, int T, int D, int accumulate_dw,
                                          cudaStream_t st) {
  if (T <= 0 || D <= 0 || dy == nullptr || x == nullptr || w == nullptr || rstd == nullptr || dx == nullptr ||
      dw == nullptr)
    return FTB200_E_BADARG;
  if (D % 8) return FTB200_E_ALIGN;
  if (D > 8192) return FTB200_E_TOOBIG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return FTB200_E_CUDA;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return FTB200_E_CUDA;
  const int nblk = std::min(T, sms * 2);
  if (static_cast<long long>(nblk) * D > static_cast<long long>(FTB200_NOALLOC_SCRATCH_FLOATS)) return FTB200_E_TOOBIG;
  float* scratch = g_noalloc_scratch_addr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    // one-time set-up for this device (which is current): resolve the array's device address
    float* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_scratch) != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return FTB200_E_CUDA;
    }
    g_noalloc_scratch_addr[dev].store(p, std::memory_order_release);
    scratch = p;
  }
  return launch_rmsnorm_bwd(dy, x, w, rstd, dres, dx, dw, scratch, T, D, accumulate_dw, sms, st);
}

// ---- checked-index debug build: status query and a self-test that records an out-of-range
// index without touching memory (a launch of one thread evaluating FTB_IN_RANGE(5, 4))
#ifdef FT_BOUNDS_CHECK
namespace {
__global__ void bounds_selftest_kernel(int i, int n, int* ok) { *ok = FTB_IN_RANGE(i, n) ? 1 : 0; }
}  // namespace
FTB200_API int ftb200_bounds_selftest(int i, int n, int* ok_dev, cudaStream_t st) {
  bounds_selftest_kernel<<<1, 1, 0, st>>>(i, n, ok_dev);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}
#endif
FTB_DEFINE_BOUNDS_QUERY(elementwise)
