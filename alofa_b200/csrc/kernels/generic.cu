// Kernels that take every size: the true 32-bit path of the whole model, and
// the place the bfloat16 path falls back to for shapes its fast kernels refuse.
//
// Everything accumulates in fp32 with plain FMA (no tensor cores, no TF32, no
// approximate intrinsics; this file is compiled without fast-math).  For every
// output element the order of additions is fixed by the problem sizes alone,
// never by which other rows share the launch, so a row's result does not
// depend on how a batch was put together.
//
// Arithmetic follows the reference's scalar kernels
// (src/alofa/kernels/cpu/scalar.mojo:93-470, paged.mojo:208-336,
// segments.mojo:48-130) with fp32 instead of f64 accumulators.
#include "common.cuh"
#include <type_traits>

// ---------------------------------------------------------------------------
// Embedding: out[t, :] = table[ids[t], :] widened to fp32.
// An id outside [0, vocab) writes zeros and raises the status flag.
// ---------------------------------------------------------------------------
template <typename TW>
__global__ void embed_gather_kernel(float* __restrict__ out, const TW* __restrict__ table,
                                    const int* __restrict__ ids, const int* __restrict__ src, const int* __restrict__ fed,
                                    int hidden, int vocab, int* status) {
  pdl_begin();
  const int t = blockIdx.x;
  int id = ids[t];
  if (src && src[t] >= 0) id = fed[src[t]];  // the token an earlier step sampled, still on the device
  const bool ok = id >= 0 && id < vocab;
  if (!ok && threadIdx.x == 0 && status) atomicExch(status, 1);
  const TW* row = table + (size_t)(ok ? id : 0) * hidden;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) out[(size_t)t * hidden + c] = ok ? to_f(row[c]) : 0.f;
}

// src (optional): per token, -1 to take ids[t], else the row of `fed` (tokens
// sampled by the step before, on the device) that holds the id.
ALOFA_API int alofa_embed_gather(void* out, const void* table, const int* ids, const int* src, const int* fed, int n_tokens, int hidden,
                                 int vocab, int table_bf16, int* status, cudaStream_t stream) {
  if (n_tokens <= 0) return ALOFA_OK;
  ALOFA_PREFER_MAX_SHARED(embed_gather_kernel<bf16>);
  ALOFA_PREFER_MAX_SHARED(embed_gather_kernel<float>);
  if (table_bf16)
    launch_dep(embed_gather_kernel<bf16>, n_tokens, 256, 0, stream, (float*)out, (const bf16*)table, ids, src, fed, hidden, vocab, status);
  else
    launch_dep(embed_gather_kernel<float>, n_tokens, 256, 0, stream, (float*)out, (const float*)table, ids, src, fed, hidden, vocab, status);
  return launch_status();
}

// ---------------------------------------------------------------------------
// RMSNorm: y = x * (1/sqrt(mean(x^2) + eps)) * w, one block per output row.
// `rows` (optional) picks the input row of each output row.  With `shift`
// (optional) the layer norm instead: y = (x - mean) / sqrt(variance + eps) * w +
// shift, the variance being the mean of the squared deviations.
// ---------------------------------------------------------------------------
template <typename TO>
__global__ void rmsnorm_kernel(TO* __restrict__ out, const float* x, const float* __restrict__ w,
                               const float* __restrict__ shift, const int* __restrict__ rows, int hidden, float eps) {
  __shared__ float scratch[32];
  pdl_begin();
  const int r = blockIdx.x;
  const float* xr = x + (size_t)(rows ? rows[r] : r) * hidden;
  float mean = 0.f;
  if (shift) {
    for (int c = threadIdx.x; c < hidden; c += blockDim.x) mean += xr[c];
    mean = block_sum(mean, scratch) / (float)hidden;
  }
  float ss = 0.f;
  for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
    const float v = xr[c] - mean;
    ss = fmaf(v, v, ss);
  }
  ss = block_sum(ss, scratch);
  const float scale = 1.0f / sqrtf(ss / (float)hidden + eps);
  if (shift) for (int c = threadIdx.x; c < hidden; c += blockDim.x) out[(size_t)r * hidden + c] = from_f<TO>((xr[c] - mean) * scale * w[c] + shift[c]);
  else for (int c = threadIdx.x; c < hidden; c += blockDim.x) out[(size_t)r * hidden + c] = from_f<TO>(xr[c] * scale * w[c]);
}

// Rows of up to 4,096 numbers in whole groups of four: every load of the row is in flight at once and the row stays in
// registers, and the kernel before it may still run (one row of 896 in a decode step: 4.6 -> 1.5 us of the step's time).  A block
// has no more warps than a row has groups for them: 2,048 rows of 64 took 5.1 us with 256 threads to each, 3.1 now.
template <typename TO>
__global__ void __launch_bounds__(256) rmsnorm_vector_kernel(TO* __restrict__ out, const float* x, const float* __restrict__ w,
                                                             const float* __restrict__ shift, const int* __restrict__ rows, int hidden, float eps) {
  __shared__ float scratch[32];
  const int n4 = hidden >> 2, step = blockDim.x;
  float4 v[4], g[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // the norm's weight is a constant of the model: read ahead of the wait
    const int c = threadIdx.x + i * step;
    g[i] = c < n4 ? reinterpret_cast<const float4*>(w)[c] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  pdl_begin();
  const int r = blockIdx.x;
  const float4* xr = reinterpret_cast<const float4*>(x + (size_t)(rows ? rows[r] : r) * hidden);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = threadIdx.x + i * step;
    v[i] = c < n4 ? xr[c] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float mean = 0.f;
  if (shift) {
#pragma unroll
    for (int i = 0; i < 4; ++i) mean += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    mean = block_sum(mean, scratch) / (float)hidden;
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (threadIdx.x + i * step >= n4) continue;
    const float a = v[i].x - mean, b = v[i].y - mean, c = v[i].z - mean, d = v[i].w - mean;
    ss = fmaf(a, a, ss), ss = fmaf(b, b, ss), ss = fmaf(c, c, ss), ss = fmaf(d, d, ss);
  }
  ss = block_sum(ss, scratch);
  const float scale = 1.0f / sqrtf(ss / (float)hidden + eps);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = threadIdx.x + i * step;
    if (c >= n4) continue;
    float y[4] = {(v[i].x - mean) * scale * g[i].x, (v[i].y - mean) * scale * g[i].y, (v[i].z - mean) * scale * g[i].z, (v[i].w - mean) * scale * g[i].w};
    TO* o = out + (size_t)r * hidden + 4 * c;
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = from_f<TO>(shift ? y[j] + shift[4 * c + j] : y[j]);
  }
}

ALOFA_API int alofa_rmsnorm(void* out, const void* x, const void* w, const float* shift, const int* rows, int n_rows, int hidden, float eps,
                            int out_bf16, cudaStream_t stream) {
  if (n_rows <= 0) return ALOFA_OK;
  const bool vector = hidden % 4 == 0 && hidden <= 4096 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
  const int threads = vector && hidden > 0 && hidden < 1024 ? (hidden / 4 + 31) / 32 * 32 : 256;
  if (out_bf16)
    launch_dep(vector ? rmsnorm_vector_kernel<bf16> : rmsnorm_kernel<bf16>, n_rows, threads, 0, stream, (bf16*)out, (const float*)x, (const float*)w, shift, rows, hidden, eps);
  else
    launch_dep(vector ? rmsnorm_vector_kernel<float> : rmsnorm_kernel<float>, n_rows, threads, 0, stream, (float*)out, (const float*)x, (const float*)w, shift, rows, hidden, eps);
  return launch_status();
}

// ---------------------------------------------------------------------------
// Matrix product y = x W^T (+ bias), W row-major [N, K].
//   EPI_STORE    out[m, n] = acc
//   EPI_RESIDUAL out[m, n] += acc        (out is the fp32 residual stream)
//   EPI_GATED    W holds [gate; up] (2N rows): out[m, n] = silu(gate) * up, or the clamped form of gate_times
// EPI_STORE | (code << 4): out[m, n] = act(acc + bias), the activation codes of common.cuh.
// 64x64 tile, 16-deep slices, 256 threads with 4x4 outputs each; every output
// is summed by one thread over k ascending.
// ---------------------------------------------------------------------------
enum { EPI_STORE = 0, EPI_RESIDUAL = 1, EPI_GATED = 2 };

template <typename TA, typename TW, typename TO, int EPI>
__global__ void __launch_bounds__(256) gemm_generic_kernel(TO* __restrict__ out, const TA* __restrict__ x,
                                                           const TW* __restrict__ w, const float* __restrict__ bias, int M,
                                                           int N, int K, int act, float gate_alpha, float gate_limit) {
  constexpr int BM = 64, BN = 64, BK = 16;
  constexpr int NW = (EPI == EPI_GATED) ? 2 : 1;
  __shared__ float xs[BK][BM + 1];
  __shared__ float ws[NW][BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[NW][4][4];
#pragma unroll
  for (int a = 0; a < NW; ++a)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[a][i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + 256 * i;
      const int r = e >> 4, k = e & 15;
      const int gm = m0 + r, gk = k0 + k;
      xs[k][r] = (gm < M && gk < K) ? to_f(x[(size_t)gm * K + gk]) : 0.f;
      const int gn = n0 + r;
#pragma unroll
      for (int a = 0; a < NW; ++a)
        ws[a][k][r] = (gn < N && gk < K) ? to_f(w[((size_t)a * N + gn) * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float xv[4], wv[NW][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) xv[i] = xs[k][ty + 16 * i];
#pragma unroll
      for (int a = 0; a < NW; ++a)
#pragma unroll
        for (int j = 0; j < 4; ++j) wv[a][j] = ws[a][k][tx + 16 * j];
#pragma unroll
      for (int a = 0; a < NW; ++a)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[a][i][j] = fmaf(xv[i], wv[a][j], acc[a][i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx + 16 * j;
      if (gn >= N) continue;
      const size_t o = (size_t)gm * N + gn;
      if (EPI == EPI_GATED) {
        float g = acc[0][i][j], u = acc[NW - 1][i][j];
        if (bias) {
          g += bias[gn];
          u += bias[N + gn];
        }
        out[o] = from_f<TO>(gate_times(g, u, gate_alpha, gate_limit));
      } else {
        float v = acc[0][i][j];
        if (bias) v += bias[gn];
        if (EPI == EPI_RESIDUAL)
          out[o] = from_f<TO>(to_f(out[o]) + v);
        else
          out[o] = from_f<TO>(activate(v, act));
      }
    }
  }
}

// The same for 32-bit operands whose depth is a multiple of four: the product of the whole 32-bit path.  A warp owns MT
// rows of x and NT columns of the output; lane l sums the depths 4 l .. 4 l + 3 of every run of 128 in ascending order, and
// the 32 lanes' sums are added pairwise, 16, 8, 4, 2, 1 lanes apart.  That order depends on the depth alone, so a row's
// result is the same in every tile shape below, whatever rows share the launch.  A decode step is bound by the weights'
// bytes: one row takes one column a warp, with up to 16 loads of 16 bytes a lane in flight and the first of them ahead of
// the dependency wait, where the 64 x 64 tiles above kept 14 of 148 SMs busy (one row, output and down projection of 896
// columns: 318 -> 3.7 us on average; gate and up 244 -> 6.5 us, 5.4 TB/s).  A few more rows are bound by the reads of x and w
// through L1: 8 x 4 sums a lane from 12 such reads (16 rows, gate and up: 22 us).
template <int V>
__device__ __forceinline__ float reduce_across_lanes(float (&v)[V], int lane) {  // value i ends in the lanes i * (32 / V) ..
  int o = 16;
#pragma unroll
  for (int half = V / 2; half >= 1; half >>= 1, o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float mine = upper ? v[half + i] : v[i], sent = upper ? v[i] : v[half + i];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, sent, o);
    }
  }
  float s = v[0];
#pragma unroll
  for (int left = 32 / V / 2; left >= 1; left >>= 1) s += __shfl_xor_sync(0xffffffffu, s, left);
  return s;
}

template <int MT, int R, int EPI>
__device__ __forceinline__ void finish_f32(const float (&acc)[MT * R], int lane, float* out, const float* __restrict__ bias, int m0, int n0, int M, int N, int act, float gate_alpha, float gate_limit) {
  constexpr int NW = EPI == EPI_GATED ? 2 : 1, V = MT * R, G = V > 32 ? 32 : V;  // values reduced together: value i of a group ends in the lanes i * (32 / G) ..
#pragma unroll
  for (int g = 0; g < V; g += G) {
    float part[G];
#pragma unroll
    for (int j = 0; j < G; ++j) part[j] = acc[g + j];
    float v = reduce_across_lanes<G>(part, lane);
    const int i = g + lane / (32 / G);  // the value this lane holds: row i / R, column (i % R) / NW, its gate or up sum
    const int m = m0 + i / R, n = n0 + (i % R) / NW;
    float u = 0.f;
    if (EPI == EPI_GATED) u = __shfl_xor_sync(0xffffffffu, v, 32 / G);  // the up sum beside the gate's
    if (m >= M || n >= N || lane % (32 / G) || (EPI == EPI_GATED && i % NW)) continue;
    float* o = out + (size_t)m * N + n;
    if (EPI == EPI_GATED) {
      if (bias) v += bias[n], u += bias[N + n];
      *o = gate_times(v, u, gate_alpha, gate_limit);
    } else {
      if (bias) v += bias[n];
      *o = EPI == EPI_RESIDUAL ? *o + v : activate(v, act);
    }
  }
}

template <int MT, int NT, int EPI>
__global__ void __launch_bounds__(256) gemm_f32_kernel(float* out, const float* x, const float* __restrict__ w, const float* __restrict__ bias, int M, int N, int K, int act,
                                                       float gate_alpha, float gate_limit) {
  constexpr int NW = EPI == EPI_GATED ? 2 : 1, R = NT * NW, V = MT * R;
  constexpr int U = V == 1 ? 16 : R >= 8 ? 1 : 8 / R;  // runs of 128 whose weights are asked for together
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 8 + warp) * NT, m0 = blockIdx.y * MT;
  const int k4 = K >> 2;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4* wr[R];  // columns past the last read the last one's weights, and are not stored
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = reinterpret_cast<const float4*>(w + ((size_t)(r % NW) * N + min(n0 + r / NW, N - 1)) * K);
  float4 wv[U][R];
  auto load_weights = [&](int c) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) wv[u][r] = c + u * 32 < k4 ? __ldg(wr[r] + c + u * 32) : zero;
  };
  load_weights(lane);
  pdl_begin();
  const float4* xr[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) xr[m] = reinterpret_cast<const float4*>(x + (size_t)min(m0 + m, M - 1) * K);
  float acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.f;
  for (int c = lane; c < k4; c += 32 * U) {  // a lane past the end has left the loop: its sums stand
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float4 xv[MT];
#pragma unroll
      for (int m = 0; m < MT; ++m) xv[m] = c + u * 32 < k4 ? xr[m][c + u * 32] : zero;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float& a = acc[m * R + r];
          a = fmaf(xv[m].x, wv[u][r].x, a), a = fmaf(xv[m].y, wv[u][r].y, a);
          a = fmaf(xv[m].z, wv[u][r].z, a), a = fmaf(xv[m].w, wv[u][r].w, a);
        }
    }
    load_weights(c + 32 * U);
  }
  finish_f32<MT, R, EPI>(acc, lane, out, bias, m0, n0, M, N, act, gate_alpha, gate_limit);
}

// The same over prompts: blocks of 32 rows and 32 rows of the weight, a warp 16 x 8 sums a lane.  Runs of 128 numbers of the
// depth come into shared memory three deep: read straight from L2 through L1, the rows of x stood in the way of 512
// multiply-adds a lane and run, and what two warps a scheduler could not hide made long prompts slower than the 64 x 64 tiles
// above (2,048 rows, gate and up of the 0.5B shape: 1,392 us there, 1,627 straight from L2, now 1,212; output head, 40 rows 683,
// 787 and 575).  Depths a little over a run or two leave lanes idle: from 4,096 rows on the tiles, whose order of summation is another
// one, are still faster at depth 260 (x 257, gated: 72 us there, 82 here).
constexpr int F32_ROWS = 32, F32_WEIGHT_ROWS = 32, F32_STAGES = 3;
constexpr size_t F32_SMEM = (size_t)F32_STAGES * (F32_ROWS + F32_WEIGHT_ROWS) * 128 * sizeof(float);
__device__ __forceinline__ void fetch16(float4* to, const float4* from, bool there) {  // zeros where nothing is there
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(there ? 16 : 0) : "memory");
}

template <int EPI>
__global__ void __launch_bounds__(256) gemm_f32_prompt_kernel(float* out, const float* x, const float* __restrict__ w, const float* __restrict__ bias, int M, int N, int K, int act,
                                                              float gate_alpha, float gate_limit) {
  constexpr int NW = EPI == EPI_GATED ? 2 : 1, MT = 16, R = 8, NT = R / NW;
  extern __shared__ float4 stages[];  // [stage][rows of x, rows of the weight][lane]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.y * F32_ROWS, column0 = blockIdx.x * (F32_WEIGHT_ROWS / NW);
  const int k4 = K >> 2, runs = (k4 + 31) >> 5;
  // this warp fetches every eighth row of both; rows and columns past the last read the last one's, and are not stored
  const float4 *wr[4], *xr[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp + 8 * i;
    wr[i] = reinterpret_cast<const float4*>(w + ((size_t)(r % NW) * N + min(column0 + r / NW, N - 1)) * K);
    xr[i] = reinterpret_cast<const float4*>(x + (size_t)min(row0 + r, M - 1) * K);
  }
  auto stage = [&](int run) { return stages + (size_t)(run % F32_STAGES) * (F32_ROWS + F32_WEIGHT_ROWS) * 32; };
  auto fetch = [&](const float4* const (&rows)[4], int run, int to) {
    const int c = run * 32 + lane;
#pragma unroll
    for (int i = 0; i < 4; ++i) fetch16(stage(run) + (to + warp + 8 * i) * 32 + lane, rows[i] + (c < k4 ? c : 0), c < k4);
  };
#pragma unroll
  for (int run = 0; run < F32_STAGES - 1; ++run)
    if (run < runs) fetch(wr, run, F32_ROWS);
  pdl_begin();
#pragma unroll
  for (int run = 0; run < F32_STAGES - 1; ++run) {
    if (run < runs) fetch(xr, run, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[MT * R];
#pragma unroll
  for (int v = 0; v < MT * R; ++v) acc[v] = 0.f;
  const int mine = (warp % 2) * MT, theirs = F32_ROWS + (warp / 2) * R;  // this warp's rows of x and of the weight
  for (int run = 0; run < runs; ++run) {
    asm volatile("cp.async.wait_group %0;" ::"n"(F32_STAGES - 2) : "memory");
    __syncthreads();  // the run is here, and every warp is done with the one whose stage is fetched into next
    if (run + F32_STAGES - 1 < runs) fetch(wr, run + F32_STAGES - 1, F32_ROWS), fetch(xr, run + F32_STAGES - 1, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float4* here = stage(run) + lane;
    float4 wv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) wv[r] = here[(theirs + r) * 32];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float4 xv = here[(mine + m) * 32];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float& a = acc[m * R + r];
        a = fmaf(xv.x, wv[r].x, a), a = fmaf(xv.y, wv[r].y, a), a = fmaf(xv.z, wv[r].z, a), a = fmaf(xv.w, wv[r].w, a);
      }
    }
  }
  finish_f32<MT, R, EPI>(acc, lane, out, bias, row0 + mine, column0 + (warp / 2) * NT, M, N, act, gate_alpha, gate_limit);
}

// The pairwise sum of COUNT lanes' products, STRIDE apart from lane l on: 4 rows of x 16 apart by 4 rows of the weight 16 apart.
template <int COUNT, int STRIDE, int PITCH>
struct LaneSums {
  __device__ static __forceinline__ void of(float (&s)[16], const float4* xs, const float4* ws, int l) {
    float t[16];
    LaneSums<COUNT / 2, STRIDE * 2, PITCH>::of(s, xs, ws, l);
    LaneSums<COUNT / 2, STRIDE * 2, PITCH>::of(t, xs, ws, l + STRIDE);
#pragma unroll
    for (int v = 0; v < 16; ++v) s[v] += t[v];
  }
};
template <int STRIDE, int PITCH>
struct LaneSums<1, STRIDE, PITCH> {
  __device__ static __forceinline__ void of(float (&s)[16], const float4* xs, const float4* ws, int l) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = xs[16 * i * PITCH + l], b[i] = ws[16 * i * PITCH + l];
#pragma unroll
    for (int v = 0; v < 16; ++v) {
      const float4 p = a[v >> 2], q = b[v & 3];
      s[v] = fmaf(p.w, q.w, fmaf(p.z, q.z, fmaf(p.y, q.y, fmaf(p.x, q.x, 0.f))));
    }
  }
};

// The same for depths of up to 4 GROUPS over many rows: blocks of 64 rows and 64 rows of the weight, whole in shared memory, a thread
// 4 x 4 sums of its own.  What lane l would sum is summed for one l after the other, in the order in which the pairwise sums close:
// 0 and half of the lanes on, a quarter on and three quarters on, and so forth.  (With the depth over the lanes a depth of 16 leaves 28
// of 32 idle and a block has little to do between its start and its end: 2,048 rows x 2,048 of depth 16 79 us, here 10.6, and 10.1 in
// the 64 x 64 tiles further up.)
template <int EPI, int GROUPS>
__global__ void __launch_bounds__(256, 2) gemm_f32_short_kernel(float* out, const float* x, const float* __restrict__ w, const float* __restrict__ bias, int M, int N, int K, int act,
                                                                float gate_alpha, float gate_limit) {
  constexpr int NW = EPI == EPI_GATED ? 2 : 1, COLUMNS = 64 / NW, PITCH = GROUPS + 1;  // odd: eight neighbouring rows lie in different banks
  extern __shared__ float4 stages[];  // 64 rows of x, 64 of the weight (gated: 32 columns' gate rows, then their up rows)
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int row0 = blockIdx.y * 64, column0 = blockIdx.x * COLUMNS, k4 = K >> 2;
  const float4 *xs = stages + ty * PITCH, *ws = stages + (64 + tx) * PITCH;
#pragma unroll
  for (int i = threadIdx.x; i < 64 * GROUPS; i += 256) {  // rows and columns past the last read the last one's, and are not stored
    const int r = i / GROUPS, c = i % GROUPS;
    const float4* row = reinterpret_cast<const float4*>(w + ((size_t)(r / COLUMNS) * N + min(column0 + r % COLUMNS, N - 1)) * K);
    fetch16(stages + (64 + r) * PITCH + c, row + min(c, k4 - 1), c < k4);
  }
  pdl_begin();
#pragma unroll
  for (int i = threadIdx.x; i < 64 * GROUPS; i += 256) {
    const int r = i / GROUPS, c = i % GROUPS;
    fetch16(stages + r * PITCH + c, reinterpret_cast<const float4*>(x + (size_t)min(row0 + r, M - 1) * K) + min(c, k4 - 1), c < k4);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float acc[16];
  LaneSums<GROUPS, 1, PITCH>::of(acc, xs, ws, 0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = row0 + ty + 16 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4 / NW; ++j) {
      const int n = column0 + tx + 16 * j;
      if (n >= N) continue;
      float* o = out + (size_t)m * N + n;
      float v = acc[4 * i + j];
      if (EPI == EPI_GATED) {
        float u = acc[4 * i + j + 2];
        if (bias) v += bias[n], u += bias[N + n];
        *o = gate_times(v, u, gate_alpha, gate_limit);
      } else {
        if (bias) v += bias[n];
        *o = EPI == EPI_RESIDUAL ? *o + v : activate(v, act);
      }
    }
  }
}

template <int EPI>
static int gemm_f32_launch(float* out, const float* x, const float* w, const float* bias, int M, int N, int K, int act, float gate_alpha, float gate_limit, cudaStream_t stream) {
  constexpr int NW = EPI == EPI_GATED ? 2 : 1;
  auto launch = [&](auto kernel, int mt, int columns, size_t smem) {
    const long long rows = (M + mt - 1) / mt;
    if (rows > 65535) return ALOFA_ERR_ARGUMENT;
    launch_dep(kernel, dim3((N + columns - 1) / columns, (unsigned)rows), 256, smem, stream, out, x, w, bias, M, N, K, act, gate_alpha, gate_limit);
    return launch_status();
  };
  if (M == 1) return launch(gemm_f32_kernel<1, 1, EPI>, 1, 8, 0);
  if (M == 2) return launch(gemm_f32_kernel<2, 2 / NW, EPI>, 2, 16 / NW, 0);
  if (M <= 4) return launch(gemm_f32_kernel<4, 2 / NW, EPI>, 4, 16 / NW, 0);
  static int sms = 0;
  if (!sms) {
    int device = 0, count = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_f32_prompt_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F32_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_f32_short_kernel<EPI, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(128 * 33 * sizeof(float4))) != cudaSuccess)
      return ALOFA_ERR_LAUNCH;
    sms = count;
  }
  // Blocks of 32 rows once they come to half of the SMs and most of the rows are there (us with 8 x 4 sums a warp / in such blocks:
  // depth 896 x 4,864 gated 16 rows 22.3 / 29.5, 24 rows 30.7 / 29.0; depth 4,864 x 896, 28 column blocks, 64 rows 38.5 / 40.6, 96
  // rows 56.5 / 41.6; depth 896 x 1,152, 64 rows 10.3 / 9.6).
  const int columns = F32_WEIGHT_ROWS / NW;
  const long long blocks = (long long)((N + columns - 1) / columns) * ((M + F32_ROWS - 1) / F32_ROWS);
  if (M > 16 && 2 * blocks >= sms) {
    // Short depths: blocks of 64 rows, at depths of more than 32 once they too come to half of the SMs (us in blocks of 32 / of 64:
    // depth 16 x 2,048 40 rows 6.0 / 3.5, 2,048 rows 79 / 10.6; depth 128 x 128 1,024 rows 4.3 / 7.7, 4,096 rows 12.6 / 9.0).
    const long long blocks64 = (long long)((N + 64 / NW - 1) / (64 / NW)) * ((M + 63) / 64);
    if (K > 128 || K == 0 || (K > 32 && 2 * blocks64 < sms)) return launch(gemm_f32_prompt_kernel<EPI>, F32_ROWS, columns, F32_SMEM);
    auto launch_short = [&](auto kernel, int groups) { return launch(kernel, 64, 64 / NW, (size_t)128 * (groups + 1) * sizeof(float4)); };
    if (K > 64) return launch_short(gemm_f32_short_kernel<EPI, 32>, 32);
    if (K > 32) return launch_short(gemm_f32_short_kernel<EPI, 16>, 16);
    if (K > 16) return launch_short(gemm_f32_short_kernel<EPI, 8>, 8);
    return launch_short(gemm_f32_short_kernel<EPI, 4>, 4);
  }
  return launch(gemm_f32_kernel<8, 4 / NW, EPI>, 8, 32 / NW, 0);
}

template <typename TA, typename TW, typename TO>
static int gemm_generic_launch(void* out, const void* x, const void* w, const float* bias, int M, int N, int K, int epi,
                               float gate_alpha, float gate_limit, cudaStream_t stream) {
  const int act = epi >> 4;  // EPI_STORE only: an activation on the sums (codes of common.cuh)
  epi &= 15;
  if (act && epi != EPI_STORE) return ALOFA_ERR_ARGUMENT;
  dim3 grid((N + 63) / 64, (M + 63) / 64);
  if (epi == EPI_STORE)
    gemm_generic_kernel<TA, TW, TO, EPI_STORE><<<grid, 256, 0, stream>>>((TO*)out, (const TA*)x, (const TW*)w, bias, M, N, K, act, gate_alpha, gate_limit);
  else if (epi == EPI_RESIDUAL)
    gemm_generic_kernel<TA, TW, TO, EPI_RESIDUAL><<<grid, 256, 0, stream>>>((TO*)out, (const TA*)x, (const TW*)w, bias, M, N, K, act, gate_alpha, gate_limit);
  else if (epi == EPI_GATED)
    gemm_generic_kernel<TA, TW, TO, EPI_GATED><<<grid, 256, 0, stream>>>((TO*)out, (const TA*)x, (const TW*)w, bias, M, N, K, act, gate_alpha, gate_limit);
  else
    return ALOFA_ERR_ARGUMENT;
  return launch_status();
}

// dtype flags: 0 = fp32, 1 = bf16.  N is the number of output columns (for
// EPI_GATED the weight has 2N rows).  EPI_RESIDUAL requires an fp32 output.
ALOFA_API int alofa_gemm_generic(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int epi,
                                 int x_bf16, int w_bf16, int out_bf16, float gate_alpha, float gate_limit, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return ALOFA_OK;
  if (K <= 0) return ALOFA_ERR_ARGUMENT;
  if ((epi & 15) == EPI_RESIDUAL && out_bf16) return ALOFA_ERR_ARGUMENT;
  const float* b = (const float*)bias;
  const int key = (x_bf16 ? 4 : 0) | (w_bf16 ? 2 : 0) | (out_bf16 ? 1 : 0);
  switch (key) {
    case 0:
      if (K % 4 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0 && M <= 8 * 65535) {  // rows of whole groups of 16 bytes
        const int act = epi >> 4;
        if (act && (epi & 15) != EPI_STORE) return ALOFA_ERR_ARGUMENT;
        switch (epi & 15) {
          case EPI_STORE: return gemm_f32_launch<EPI_STORE>((float*)out, (const float*)x, (const float*)w, b, M, N, K, act, gate_alpha, gate_limit, stream);
          case EPI_RESIDUAL: return gemm_f32_launch<EPI_RESIDUAL>((float*)out, (const float*)x, (const float*)w, b, M, N, K, act, gate_alpha, gate_limit, stream);
          case EPI_GATED: return gemm_f32_launch<EPI_GATED>((float*)out, (const float*)x, (const float*)w, b, M, N, K, act, gate_alpha, gate_limit, stream);
          default: return ALOFA_ERR_ARGUMENT;
        }
      }
      return gemm_generic_launch<float, float, float>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    case 1: return gemm_generic_launch<float, float, bf16>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    case 2: return gemm_generic_launch<float, bf16, float>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    case 3: return gemm_generic_launch<float, bf16, bf16>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    case 4: return gemm_generic_launch<bf16, float, float>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    case 5: return gemm_generic_launch<bf16, float, bf16>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    case 6: return gemm_generic_launch<bf16, bf16, float>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
    default: return gemm_generic_launch<bf16, bf16, bf16>(out, x, w, b, M, N, K, epi, gate_alpha, gate_limit, stream);
  }
}

// ---------------------------------------------------------------------------
// Rotary position encoding (NeoX halves) on q and k, and the cache write.
//   qkv     [T, (nh + 2 nkv) * hd]  q heads, then k heads, then v heads
//   q_out   [T, nh * hd]            rotated queries
//   k_cache, v_cache [slots, nkv, hd]; slot_map[t] is the physical slot of
//   token t (page * page_size + offset), or < 0 to write nothing.
//   cos_sin [max_pos, rot/2, 2] fp32 (cos, sin).  rot == 0: no rotation.
// y[d] = a cos - b sin, y[d + rot/2] = b cos + a sin, a = x[d], b = x[d + rot/2];
// dims >= rot pass through.  The products are fp32.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void rope_store_kernel(T* __restrict__ q_out, T* __restrict__ k_cache, T* __restrict__ v_cache,
                                  const T* qkv, const float* __restrict__ cos_sin,
                                  const int* __restrict__ positions, const int* __restrict__ slot_map, int nh, int nkv,
                                  int hd, int rot, int write_cache) {
  pdl_begin();
  const int t = blockIdx.x;
  const int head = blockIdx.y;  // 0..nh-1 q, nh..nh+nkv-1 k, then v
  const int pos = positions[t];
  const int half = rot >> 1;
  const T* src = qkv + ((size_t)t * (nh + 2 * nkv) + head) * hd;
  T* dst;
  bool rotate = true;
  if (head < nh) {
    dst = q_out + ((size_t)t * nh + head) * hd;
  } else {
    if (!write_cache) return;
    const int slot = slot_map[t];
    if (slot < 0) return;
    if (head < nh + nkv) {
      dst = k_cache + ((size_t)slot * nkv + (head - nh)) * hd;
    } else {
      dst = v_cache + ((size_t)slot * nkv + (head - nh - nkv)) * hd;
      rotate = false;
    }
  }
  const float* cs = cos_sin + (size_t)pos * rot;  // rot/2 pairs
  for (int d = threadIdx.x; d < hd; d += blockDim.x) {
    float y;
    if (rotate && d < rot) {
      const int i = d < half ? d : d - half;
      const float c = cs[2 * i], s = cs[2 * i + 1];
      const float a = to_f(src[i]), b = to_f(src[i + half]);
      y = d < half ? (a * c - b * s) : (b * c + a * s);
    } else {
      y = to_f(src[d]);
    }
    dst[d] = from_f<T>(y);
  }
}

ALOFA_API int alofa_rope_store(void* q_out, void* k_cache, void* v_cache, const void* qkv, const float* cos_sin,
                               const int* positions, const int* slot_map, int n_tokens, int nh, int nkv, int hd, int rot,
                               int write_cache, int is_bf16, cudaStream_t stream) {
  if (n_tokens <= 0) return ALOFA_OK;
  if (rot < 0 || rot > hd || (rot & 1)) return ALOFA_ERR_ARGUMENT;
  dim3 grid(n_tokens, nh + 2 * nkv);
  const int threads = hd <= 32 ? 32 : (hd <= 64 ? 64 : 128);
  if (is_bf16)
    launch_dep(rope_store_kernel<bf16>, grid, threads, 0, stream, (bf16*)q_out, (bf16*)k_cache, (bf16*)v_cache, (const bf16*)qkv,
               cos_sin, positions, slot_map, nh, nkv, hd, rot, write_cache);
  else
    launch_dep(rope_store_kernel<float>, grid, threads, 0, stream, (float*)q_out, (float*)k_cache, (float*)v_cache, (const float*)qkv,
               cos_sin, positions, slot_map, nh, nkv, hd, rot, write_cache);
  return launch_status();
}

// ---------------------------------------------------------------------------
// Causal grouped-query attention over the paged cache, one block per
// (token, query head).  The query at position P of request r sees the keys
// max(0, P - window + 1) .. P (window <= 0: all), found through
// block_table[r][j / page_size].  Keys are taken in chunks of 128 whose
// boundaries depend on the key index only; within a chunk each thread scores
// one key, the block takes max and sum in a fixed order, and the value sum is
// rescaled as in streaming softmax.  score = dot * scale, then (softcap > 0)
// softcap * tanh(score / softcap), all in fp32.  Keys have hd numbers per head,
// values vd (the two caches have their own row widths); v_share neighbouring key heads read one value
// head; chunk > 0: a query sees only the keys of its own chunk of that many positions.  keep > 0: keys j < keep are
// seen beside the window.  slopes: slopes[h] * (P - j) is taken off the score (after scale and cap).
// ---------------------------------------------------------------------------
template <typename T, typename TO>
__global__ void __launch_bounds__(128) paged_attention_generic_kernel(
    TO* __restrict__ out, const T* q, const T* k_cache, const T* v_cache,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table,
    int max_blocks, int page_size, int nh, int nkv, int hd, int vd, int window, float scale, float softcap, const float* __restrict__ sink,
    int chunk, int v_share, int keep, const float* __restrict__ slopes) {
  extern __shared__ __align__(16) float smem[];
  pdl_begin();
  float* qs = smem;          // hd
  float* ps = smem + hd;     // 128
  __shared__ float scratch[32];
  __shared__ int pages[128];
  const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int kvh = h / (nh / nkv);
  const int P = positions[t];
  const int* table = block_table + (size_t)seq_of_token[t] * max_blocks;
  for (int d = tid; d < hd; d += 128) qs[d] = to_f(q[((size_t)t * nh + h) * hd + d]);
  int first = 0;
  if (window > 0 && P - window + 1 > 0) first = P - window + 1;
  if (chunk > 0) first = max(first, P - P % chunk);  // chunks are counted from the sequence's position 0
  const int vh = kvh / v_share, nv = nkv / v_share;  // v_share neighbouring key heads read one value head
  // a sink is one more term of the softmax's denominator, exp(sink[h]), that belongs to no key and has no value
  float m = sink ? sink[h] : -INFINITY, l = sink ? 1.f : 0.f;
  float acc0 = 0.f, acc1 = 0.f;  // dims tid and tid + 128
  const int kept = min(keep, first);  // keys [0, kept) and [first, P] are seen
  const float slope = slopes ? slopes[h] : 0.f;
  __syncthreads();
  for (int c0 = kept > 0 ? 0 : (first / 128) * 128; c0 <= P; c0 += 128) {
    if (c0 >= kept) c0 = max(c0, (first / 128) * 128);  // nothing between the kept keys and the window
    const int j = c0 + tid;
    const bool visible = (j >= first || j < kept) && j <= P;
    float s = -INFINITY;
    int slot = -1;
    if (visible) {
      const int page = table[j / page_size];
      slot = page * page_size + (j % page_size);
      const T* kr = k_cache + ((size_t)slot * nkv + kvh) * hd;
      float dot = 0.f;
      for (int d = 0; d < hd; ++d) dot = fmaf(qs[d], to_f(kr[d]), dot);
      s = dot * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      s -= slope * (float)(P - j);
    }
    pages[tid] = slot;
    const float cmax = block_max(s, scratch);
    const float m_new = fmaxf(m, cmax);
    const float p = visible ? expf(s - m_new) : 0.f;
    ps[tid] = p;
    const float csum = block_sum(p, scratch);  // also orders the writes of ps / pages
    const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
    l = l * corr + csum;
    acc0 *= corr;
    acc1 *= corr;
    const int n_in = min(128, P - c0 + 1);
    for (int i = 0; i < n_in; ++i) {
      const int sl = pages[i];
      if (sl < 0) continue;
      const T* vr = v_cache + ((size_t)sl * nv + vh) * vd;
      const float pi = ps[i];
      if (tid < vd) acc0 = fmaf(pi, to_f(vr[tid]), acc0);
      if (tid + 128 < vd) acc1 = fmaf(pi, to_f(vr[tid + 128]), acc1);
    }
    m = m_new;
    __syncthreads();
  }
  TO* o = out + ((size_t)t * nh + h) * vd;
  if (tid < vd) o[tid] = from_f<TO>(acc0 / l);
  if (tid + 128 < vd) o[tid + 128] = from_f<TO>(acc1 / l);
}

// The same where keys and values are whole groups of four numbers: a key's row is read four numbers at a time, all of it in
// flight at once, and the value sum is spread over all 128 threads, a group of vd / 4 threads taking every G-th key of a chunk;
// the groups' sums are added in order at the end.  Chunks and the order within one go by the key's index alone, as above.
// A block's time is its dependent trips to memory (one row of 14 heads over 48 keys: 21 -> 8.8 us).
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

template <typename T, typename TO>
__global__ void __launch_bounds__(128) paged_attention_vector_kernel(
    TO* __restrict__ out, const T* q, const T* k_cache, const T* v_cache,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table,
    int max_blocks, int page_size, int nh, int nkv, int hd, int vd, int window, float scale, float softcap, const float* __restrict__ sink,
    int chunk, int v_share, int keep, const float* __restrict__ slopes) {
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;            // hd
  float* ps = qs + hd;         // 128
  float* sums = ps + 128;      // [G][vd], at most 512
  __shared__ float scratch[32];
  __shared__ int pages[128];
  pdl_begin();
  const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int kvh = h / (nh / nkv);
  const int P = positions[t];
  const int* table = block_table + (size_t)seq_of_token[t] * max_blocks;
  for (int d = tid; d < hd; d += 128) qs[d] = to_f(q[((size_t)t * nh + h) * hd + d]);
  int first = 0;
  if (window > 0 && P - window + 1 > 0) first = P - window + 1;
  if (chunk > 0) first = max(first, P - P % chunk);
  const int vh = kvh / v_share, nv = nkv / v_share;
  float m = sink ? sink[h] : -INFINITY, l = sink ? 1.f : 0.f;
  const int nd = vd >> 2, G = 128 / nd;
  const int grp = tid / nd, d4 = tid - grp * nd;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  const int kept = min(keep, first);
  const float slope = slopes ? slopes[h] : 0.f;
  __syncthreads();
  for (int c0 = kept > 0 ? 0 : (first / 128) * 128; c0 <= P; c0 += 128) {
    if (c0 >= kept) c0 = max(c0, (first / 128) * 128);
    const int j = c0 + tid;
    const bool visible = (j >= first || j < kept) && j <= P;
    float s = -INFINITY;
    int slot = -1;
    if (visible) {
      const int page = table[j / page_size];
      slot = page * page_size + (j % page_size);
      const T* kr = k_cache + ((size_t)slot * nkv + kvh) * hd;
      float4 dot = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 16
      for (int d = 0; d < hd; d += 4) {
        const float4 a = load4(kr + d), b = *reinterpret_cast<const float4*>(qs + d);
        dot.x = fmaf(b.x, a.x, dot.x), dot.y = fmaf(b.y, a.y, dot.y), dot.z = fmaf(b.z, a.z, dot.z), dot.w = fmaf(b.w, a.w, dot.w);
      }
      s = ((dot.x + dot.y) + (dot.z + dot.w)) * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      s -= slope * (float)(P - j);
    }
    pages[tid] = slot;
    const float cmax = block_max(s, scratch);
    const float m_new = fmaxf(m, cmax);
    const float p = visible ? expf(s - m_new) : 0.f;
    ps[tid] = p;
    const float csum = block_sum(p, scratch);  // also orders the writes of ps / pages
    const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
    l = l * corr + csum;
    acc.x *= corr, acc.y *= corr, acc.z *= corr, acc.w *= corr;
    const int n_in = min(128, P - c0 + 1);
    if (grp < G) {
#pragma unroll 8
      for (int i = grp; i < n_in; i += G) {
        const int sl = pages[i];
        const float4 v = sl >= 0 ? load4(v_cache + ((size_t)sl * nv + vh) * vd + 4 * d4) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float pi = ps[i];
        acc.x = fmaf(pi, v.x, acc.x), acc.y = fmaf(pi, v.y, acc.y), acc.z = fmaf(pi, v.z, acc.z), acc.w = fmaf(pi, v.w, acc.w);
      }
    }
    m = m_new;
    __syncthreads();
  }
  if (grp < G) *reinterpret_cast<float4*>(sums + grp * vd + 4 * d4) = acc;
  __syncthreads();
  TO* o = out + ((size_t)t * nh + h) * vd;
  for (int d = tid; d < vd; d += 128) {
    float total = 0.f;
    for (int g = 0; g < G; ++g) total += sums[g * vd + d];
    o[d] = from_f<TO>(total / l);
  }
}

ALOFA_API int alofa_paged_attention_generic(void* out, const void* q, const void* k_cache, const void* v_cache,
                                            const int* positions, const int* seq_of_token, const int* block_table,
                                            int max_blocks, int page_size, int n_tokens, int nh, int nkv, int hd,
                                            int vd, int window, float scale, float softcap, const float* sink, int is_bf16, int chunk, int v_share,
                                            int out_f32, int keep, const float* slopes, cudaStream_t stream) {
  if (n_tokens <= 0) return ALOFA_OK;
  if (hd <= 0 || vd <= 0 || vd > 256 || nkv <= 0 || nh % nkv != 0 || page_size <= 0 || chunk < 0 || v_share <= 0 || nkv % v_share != 0 || keep < 0) return ALOFA_ERR_ARGUMENT;
  dim3 grid(n_tokens, nh);
  auto launch = [&](auto* o, const auto* queries) {
    using TO = std::remove_pointer_t<decltype(o)>;
    using T = std::remove_const_t<std::remove_pointer_t<decltype(queries)>>;
    // rows of whole groups of four numbers, which then lie on the 16 (bfloat16: 8) bytes a load takes
    bool vector = hd % 4 == 0 && vd % 4 == 0 && ((uintptr_t)k_cache | (uintptr_t)v_cache) % (4 * sizeof(T)) == 0;
    size_t smem = (size_t)(hd + 128) * sizeof(float);
    const size_t sums = vector ? (size_t)(128 / (vd / 4)) * vd * sizeof(float) : 0;
    vector = vector && smem + sums <= 47 * 1024;  // beside the static part, within what a launch has without asking for more
    if (vector) smem += sums;
    launch_dep(vector ? paged_attention_vector_kernel<T, TO> : paged_attention_generic_kernel<T, TO>, grid, 128, smem, stream,
               o, queries, (const T*)k_cache, (const T*)v_cache, positions, seq_of_token, block_table,
               max_blocks, page_size, nh, nkv, hd, vd, window, scale, softcap, sink, chunk, v_share, keep, slopes);
  };
  if (is_bf16 && out_f32) launch((float*)out, (const bf16*)q);
  else if (is_bf16) launch((bf16*)out, (const bf16*)q);
  else launch((float*)out, (const float*)q);
  return launch_status();
}
