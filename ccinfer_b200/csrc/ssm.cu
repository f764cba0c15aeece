// A selective state space mixer (the recurrent form of state-space duality): what surrounds its recurrence.
//
// The input projection's rows are laid out [z | x | B | C | dt]: a gate z and an input x of `inner` = H P channels,
// G groups of N channels each for B and C, and one step-size logit per head.  x, B and C pass a short causal
// convolution per channel (with bias) followed by silu; the step size is softplus(logit + dt_bias[h]) and the decay
// a = exp(-exp(A_log[h]) * step size).  Head h
// (with group g = h / (H / G)) then runs
//     S <- a_t S + B_t (dt_t x_t)^T        S [N, P], float, kept per request between steps
//     y_t = S^T C_t + D_h x_t
// (the recurrence itself is ccb_ssm_recurrence in delta_rule.cu).  Then y * silu(z) is cut into `parts` equal
// slices of the inner channels, every slice divided by the root of its own mean square (+ eps), and a weight per
// channel is applied.
//
//   ssm_prepare        a thread per (token, channel), or per four channels where sizes and addresses allow: convolution (earlier rows from the step or from the request's
//                      convolution state, which holds its last taps - 1 projected rows), bias, silu; float rows of x,
//                      B, C, and per (token, head) dt and a
//   conv_state_shift   a thread per (request, channel): the last taps - 1 projected rows of each request's portion
//                      become its convolution state (run after ssm_prepare has read the old one).  A request that
//                      brings ONE token is moved on by ssm_prepare itself (`shift_single`): the thread of a channel is
//                      the only one that reads that channel's state, so a decode step needs no second kernel
//   ssm_gate_norm      a block per (token, slice): (o + D x) silu(z), its root mean square, the weight
//
// Portions of prompts in the 16-bit path go through ccb_ssm_chunks (memory_chunks.cu) instead of the recurrence: for their
// rows ssm_prepare leaves B and C as two bfloat16 each and the logarithms of dt and a.
//
// Everything after the projection is float; the projection's rows and the convolution state are of the storage type.
#include "common.cuh"

using namespace ccb;

namespace {

// Where the rows from row `from` on go in place of bs, cs, dts and as: B and C as their bfloat16 values and what the
// rounding left, the logarithms of dt and of the decay.
struct SsmChunkRows {
  int from;
  __nv_bfloat16 *b_hi, *b_lo, *c_hi, *c_lo;
  float *log_a, *log_dt;
};

__device__ __forceinline__ float sigmoid_acc(float x) { return 1.f / (1.f + expf(-x)); }
// The gate in the norm of many rows: the accurate form in 32 bits; where the result is rounded to bfloat16, the fast exponential
// and division (some units of the last place of a float), an eighth of the instructions.  Rows that stay float, as those of
// the recurrence, have the accurate one.
template <typename T> __device__ __forceinline__ float silu_of(float x) { return x * sigmoid_acc(x); }
template <> __device__ __forceinline__ float silu_of<__nv_bfloat16>(float x) { return __fdividef(x, 1.f + __expf(-x)); }
template <typename T> __device__ __forceinline__ float4 silu4_of(float4 x) {
  return make_float4(silu_of<T>(x.x), silu_of<T>(x.y), silu_of<T>(x.z), silu_of<T>(x.w));
}
__device__ __forceinline__ float softplus_acc(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// proj [T, ld]: the convolved channels (x | B | C, `C` of them) start at column ox, dt at odt.
// conv_w [taps, C] (tap-major), conv_b [C]; conv_state [slots, taps - 1, C].
template <typename T>
__global__ void ssm_prepare_kernel(const T* __restrict__ proj, int ld, int ox, int odt,
                                   const float* __restrict__ conv_w, const float* __restrict__ conv_b, int taps,
                                   const T* conv_state, const float* __restrict__ A_log,
                                   const float* __restrict__ dt_bias, const int* __restrict__ entry_of_token,
                                   const int* __restrict__ cu_q, const int* __restrict__ state_slot,
                                   float* __restrict__ xs, float* __restrict__ bs, float* __restrict__ cs,
                                   float* __restrict__ dts, float* __restrict__ as, int rows, int H, int P, int G, int N,
                                   T* state_rw, int shift_single) {   // (state_rw is conv_state: no __restrict__ on either)
  ccb::pdl_begin();
  const int inner = H * P, gn = G * N;
  const int C = inner + 2 * gn;
  const int per_row = C + H;
  const size_t total = (size_t)rows * per_row;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_row), c = (int)(i - (size_t)t * per_row);
    const int e = entry_of_token[t];
    if (c >= C) {   // a head's step size and decay
      const int h = c - C;
      float dt = 0.f, a = 1.f;
      if (e >= 0) {
        dt = softplus_acc(to_f32(proj[(size_t)t * ld + odt + h]) + dt_bias[h]);
        a = expf(-expf(A_log[h]) * dt);
      }
      dts[(size_t)t * H + h] = dt;
      as[(size_t)t * H + h] = a;
      continue;
    }
    float v = 0.f;
    if (e >= 0) {
      const int r0 = cu_q[e];
      const int slot = state_slot[e];
      float acc = conv_b ? conv_b[c] : 0.f;
      for (int j = 0; j < taps; ++j) {
        const int src = t - (taps - 1) + j;   // the row this tap reads
        float u;
        if (src >= r0) u = to_f32(proj[(size_t)src * ld + ox + c]);
        else u = slot >= 0 ? to_f32(conv_state[((size_t)slot * (taps - 1) + (src - r0 + taps - 1)) * C + c]) : 0.f;
        acc = fmaf(conv_w[(size_t)j * C + c], u, acc);
      }
      v = acc * sigmoid_acc(acc);
      // a request that brings one token: this thread is the only reader of its channel's state, which it moves on
      if (shift_single && taps > 1 && slot >= 0 && cu_q[e + 1] - r0 == 1) {
        T* st = state_rw + (size_t)slot * (taps - 1) * C + c;
        for (int k = 0; k + 1 < taps - 1; ++k) st[(size_t)k * C] = st[(size_t)(k + 1) * C];
        st[(size_t)(taps - 2) * C] = proj[(size_t)t * ld + ox + c];
      }
    }
    if (c < inner) xs[(size_t)t * inner + c] = v;
    else if (c < inner + gn) bs[(size_t)t * gn + (c - inner)] = v;
    else cs[(size_t)t * gn + (c - inner - gn)] = v;
  }
}


// The same with four neighbouring channels a thread (every width, offset and row stride a multiple of 4, 16-byte
// rows): 8- or 16-byte loads of the rows, 16-byte loads of the weights and stores of the results.
template <typename T> struct In4;
template <> struct In4<float> {
  using Raw = float4;
  static __device__ __forceinline__ float4 value(const Raw a) { return a; }
  static __device__ __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
};
template <> struct In4<__nv_bfloat16> {
  using Raw = uint2;
  static __device__ __forceinline__ float4 load(const __nv_bfloat16* p) { return value(*reinterpret_cast<const uint2*>(p)); }
  static __device__ __forceinline__ float4 value(const Raw a) {
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
};

// four channels of a row to where they belong
__device__ __forceinline__ void put_channels(const float4 v, int t, int c, int inner, int gn, float* xs, float* bs, float* cs,
                                             const SsmChunkRows& chunk) {
  if (c >= inner && t >= chunk.from) {
    const bool is_b = c < inner + gn;
    const size_t at = (size_t)t * gn + (c - inner - (is_b ? 0 : gn));
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
    const float2 f0 = __bfloat1622float2(h0), f1 = __bfloat1622float2(h1);
    const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - f0.x, v.y - f0.y), l1 = __floats2bfloat162_rn(v.z - f1.x, v.w - f1.y);
    uint2 hi, lo;
    hi.x = *reinterpret_cast<const uint32_t*>(&h0);
    hi.y = *reinterpret_cast<const uint32_t*>(&h1);
    lo.x = *reinterpret_cast<const uint32_t*>(&l0);
    lo.y = *reinterpret_cast<const uint32_t*>(&l1);
    *reinterpret_cast<uint2*>((is_b ? chunk.b_hi : chunk.c_hi) + at) = hi;
    *reinterpret_cast<uint2*>((is_b ? chunk.b_lo : chunk.c_lo) + at) = lo;
    return;
  }
  float* dst = c < inner ? xs + (size_t)t * inner + c
                         : (c < inner + gn ? bs + (size_t)t * gn + (c - inner) : cs + (size_t)t * gn + (c - inner - gn));
  *reinterpret_cast<float4*>(dst) = v;
}

// a head's step size and decay
template <typename T>
__device__ __forceinline__ void put_head(const T* proj, int ld, int odt, int t, int h, int e, int H, const float* A_log,
                                         const float* dt_bias, float* dts, float* as, const SsmChunkRows& chunk) {
  float dt = 0.f, a = 1.f;
  if (e >= 0) {
    dt = softplus_acc(to_f32(proj[(size_t)t * ld + odt + h]) + dt_bias[h]);
    const float log_a = -expf(A_log[h]) * dt;
    if (t >= chunk.from) {
      chunk.log_a[(size_t)t * H + h] = log_a;
      chunk.log_dt[(size_t)t * H + h] = logf(dt);
      return;
    }
    a = expf(log_a);
  }
  dts[(size_t)t * H + h] = dt;
  as[(size_t)t * H + h] = a;
}

template <typename T>
__global__ void ssm_prepare_vec_kernel(const T* __restrict__ proj, int ld, int ox, int odt,
                                       const float* __restrict__ conv_w, const float* __restrict__ conv_b, int taps,
                                       const T* conv_state, const float* __restrict__ A_log,
                                       const float* __restrict__ dt_bias, const int* __restrict__ entry_of_token,
                                       const int* __restrict__ cu_q, const int* __restrict__ state_slot,
                                       float* __restrict__ xs, float* __restrict__ bs, float* __restrict__ cs,
                                       float* __restrict__ dts, float* __restrict__ as, int rows, int H, int P, int G,
                                       int N, T* state_rw, int shift_single, const SsmChunkRows chunk) {   // (state_rw is conv_state: no __restrict__ on either)
  ccb::pdl_begin();
  const int inner = H * P, gn = G * N;
  const int C = inner + 2 * gn;
  const int C4 = C >> 2;
  const int per_row = C4 + H;   // units of a token: groups of four channels, then one per head
  const size_t total = (size_t)rows * per_row;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_row), u4 = (int)(i - (size_t)t * per_row);
    const int e = entry_of_token[t];
    if (u4 >= C4) {
      put_head(proj, ld, odt, t, u4 - C4, e, H, A_log, dt_bias, dts, as, chunk);
      continue;
    }
    const int c = 4 * u4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (e >= 0) {
      const int r0 = cu_q[e];
      const int slot = state_slot[e];
      float4 acc = conv_b ? *reinterpret_cast<const float4*>(conv_b + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      for (int j = 0; j < taps; ++j) {
        const int src = t - (taps - 1) + j;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        if (src >= r0) u = In4<T>::load(proj + (size_t)src * ld + ox + c);
        else if (slot >= 0) u = In4<T>::load(conv_state + ((size_t)slot * (taps - 1) + (src - r0 + taps - 1)) * C + c);
        const float4 wj = *reinterpret_cast<const float4*>(conv_w + (size_t)j * C + c);
        acc.x = fmaf(wj.x, u.x, acc.x);
        acc.y = fmaf(wj.y, u.y, acc.y);
        acc.z = fmaf(wj.z, u.z, acc.z);
        acc.w = fmaf(wj.w, u.w, acc.w);
      }
      v = make_float4(acc.x * sigmoid_acc(acc.x), acc.y * sigmoid_acc(acc.y), acc.z * sigmoid_acc(acc.z),
                      acc.w * sigmoid_acc(acc.w));
      if (shift_single && taps > 1 && slot >= 0 && cu_q[e + 1] - r0 == 1) {   // (as in the kernel above)
        T* st = state_rw + (size_t)slot * (taps - 1) * C + c;
        for (int k = 0; k + 1 < taps - 1; ++k)
          for (int x = 0; x < 4; ++x) st[(size_t)k * C + x] = st[(size_t)(k + 1) * C + x];
        for (int x = 0; x < 4; ++x) st[(size_t)(taps - 2) * C + x] = proj[(size_t)t * ld + ox + c + x];
      }
    }
    put_channels(v, t, c, inner, gn, xs, bs, cs, chunk);
  }
}

// The same for steps of many rows: a thread takes its four channels (or its head) through kSsmRun neighbouring rows.  The taps'
// weights are loaded once for all of them, a row once for all the taps it meets, all loads are in flight together, and no
// thread divides to find its place.  TAPS taps.  2,048 rows of 10,240 channels with four taps, 150 MB: 90 us a row a
// thread, 60 us so (with the fast exponential 46, but its rows go into a float memory).
constexpr int kSsmRun = 4;
// from here on, rows times (groups of four channels and heads): before that a row a thread has more loads under way (10,240 channels
// and 128 heads, with 20 us of launch, a row / four rows a thread: 128 rows 28.5 / 29.9 us, 256 34.5 / 34.6, 512 45 / 38)
constexpr long long kSsmRunUnits = 1000000;
template <typename T, int TAPS>
__global__ void __launch_bounds__(256)
ssm_prepare_run_kernel(const T* __restrict__ proj, int ld, int ox, int odt, const float* __restrict__ conv_w,
                       const float* __restrict__ conv_b, const T* conv_state, const float* __restrict__ A_log,
                       const float* __restrict__ dt_bias, const int* __restrict__ entry_of_token,
                       const int* __restrict__ cu_q, const int* __restrict__ state_slot, float* __restrict__ xs,
                       float* __restrict__ bs, float* __restrict__ cs, float* __restrict__ dts, float* __restrict__ as, int rows,
                       int H, int P, int G, int N, T* state_rw, int shift_single, const SsmChunkRows chunk) {
  ccb::pdl_begin();
  __shared__ int s_entry[kSsmRun], s_back[kSsmRun], s_slot[kSsmRun], s_single[kSsmRun];
  const int inner = H * P, gn = G * N, C = inner + 2 * gn, C4 = C >> 2;
  const int t0 = blockIdx.y * kSsmRun, u4 = blockIdx.x * blockDim.x + threadIdx.x;
  if (threadIdx.x < kSsmRun) {   // of each row: its request, rows of the request before it, slot, whether it is alone
    const int t = t0 + threadIdx.x, e = t < rows ? entry_of_token[t] : -1;
    s_entry[threadIdx.x] = e;
    s_back[threadIdx.x] = e >= 0 ? t - cu_q[e] : 0;
    s_slot[threadIdx.x] = e >= 0 ? state_slot[e] : -1;
    s_single[threadIdx.x] = e >= 0 && cu_q[e + 1] - cu_q[e] == 1;
  }
  using V = typename In4<T>::Raw;
  const int c = 4 * u4;
  V raw[kSsmRun];
  if (u4 < C4) {
#pragma unroll
    for (int r = 0; r < kSsmRun; ++r)
      raw[r] = t0 + r < rows ? *reinterpret_cast<const V*>(proj + (size_t)(t0 + r) * ld + ox + c) : V{};
  }
  __syncthreads();
  if (u4 >= C4) {
    if (u4 - C4 < H)
      for (int r = 0; r < kSsmRun && t0 + r < rows; ++r)
        put_head(proj, ld, odt, t0 + r, u4 - C4, s_entry[r], H, A_log, dt_bias, dts, as, chunk);
    return;
  }
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 bias = conv_b ? *reinterpret_cast<const float4*>(conv_b + c) : zero;
  float4 cw[TAPS], win[TAPS];   // win: the row's own input last, those before it
#pragma unroll
  for (int j = 0; j < TAPS; ++j) cw[j] = *reinterpret_cast<const float4*>(conv_w + (size_t)j * C + c);
#pragma unroll
  for (int r = 0; r < kSsmRun; ++r) {
    const int t = t0 + r, e = s_entry[r], lt = s_back[r], slot = s_slot[r];
    if (t >= rows) break;
    float4 v = zero;
    if (e >= 0) {
#pragma unroll
      for (int j = 0; j + 1 < TAPS; ++j) {
        if (r > 0 && lt > 0) {   // (the row before is the same request's)
          win[j] = win[j + 1];
          continue;
        }
        const int back = TAPS - 1 - j;
        win[j] = lt >= back ? In4<T>::load(proj + (size_t)(t - back) * ld + ox + c)
                 : slot >= 0 ? In4<T>::load(conv_state + ((size_t)slot * (TAPS - 1) + (TAPS - 1 + lt - back)) * C + c) : zero;
      }
      win[TAPS - 1] = In4<T>::value(raw[r]);
      float4 acc = bias;
#pragma unroll
      for (int j = 0; j < TAPS; ++j) {
        acc.x = fmaf(cw[j].x, win[j].x, acc.x);
        acc.y = fmaf(cw[j].y, win[j].y, acc.y);
        acc.z = fmaf(cw[j].z, win[j].z, acc.z);
        acc.w = fmaf(cw[j].w, win[j].w, acc.w);
      }
      v = make_float4(acc.x * sigmoid_acc(acc.x), acc.y * sigmoid_acc(acc.y), acc.z * sigmoid_acc(acc.z),
                      acc.w * sigmoid_acc(acc.w));
      if (shift_single && TAPS > 1 && slot >= 0 && s_single[r]) {   // (as in the kernel above)
        V* st = reinterpret_cast<V*>(state_rw + (size_t)slot * (TAPS - 1) * C + c);
        for (int k = 0; k + 1 < TAPS - 1; ++k) st[(size_t)k * C4] = st[(size_t)(k + 1) * C4];
        st[(size_t)(TAPS - 2) * C4] = raw[r];
      }
    }
    put_channels(v, t, c, inner, gn, xs, bs, cs, chunk);
  }
}

// state [slots, taps - 1, C] <- the last taps - 1 of (its old rows, then the request's rows of this step).
// A thread owns one (request, channel) and walks the state's rows upwards: row i takes what row i + n held or a row
// of the step, and the rows it still has to read lie above the ones it has written.
template <typename T>
__global__ void conv_state_shift_kernel(const T* __restrict__ rows, int ld, int taps, int C, T* __restrict__ state,
                                        const int* __restrict__ cu_q, const int* __restrict__ state_slot,
                                        int entry0, int n_entries, int n_slots) {
  ccb::pdl_begin();
  const int keep = taps - 1;
  const size_t total = (size_t)n_entries * C;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int e = entry0 + (int)(i / C), c = (int)(i % C);
    const int slot = state_slot[e];
    if (slot < 0 || slot >= n_slots) continue;
    const int r0 = cu_q[e], n = cu_q[e + 1] - r0;
    if (n <= 0) continue;
    T* st = state + (size_t)slot * keep * C + c;
    for (int k = 0; k < keep; ++k) {
      const int src = k + n - keep;   // among the step's rows if >= 0, else the old state's row k + n
      st[(size_t)k * C] = src >= 0 ? rows[(size_t)(r0 + src) * ld + c] : st[(size_t)(k + n) * C];
    }
  }
}

constexpr int kGateThreads = 256;

// y[t, slice] = v / sqrt(mean(v^2) + eps) * w with v = (o + D_h x) * silu(z); o, x float [T, inner], z in proj.
template <typename T>
__global__ void __launch_bounds__(kGateThreads)
ssm_gate_norm_kernel(T* __restrict__ y, const float* __restrict__ o, const float* __restrict__ xs,
                     const T* __restrict__ proj, int ld, int oz, const float* __restrict__ Dskip,
                     const float* __restrict__ w, int P, int inner, int parts, float eps) {
  ccb::pdl_begin();
  __shared__ float red[32];
  const int t = blockIdx.x, part = blockIdx.y;
  const int width = inner / parts;
  const int c0 = part * width;
  const float* orow = o + (size_t)t * inner;
  const float* xrow = xs + (size_t)t * inner;
  const T* zrow = proj + (size_t)t * ld + oz;
  float ss = 0.f;
  for (int i = threadIdx.x; i < width; i += kGateThreads) {
    const int c = c0 + i;
    const float z = to_f32(zrow[c]);
    const float v = fmaf(Dskip[c / P], xrow[c], orow[c]) * (z * sigmoid_acc(z));
    ss += v * v;
  }
  ss = block_sum<kGateThreads>(ss, red);
  const float inv = 1.0f / sqrtf(ss / (float)width + eps);
  for (int i = threadIdx.x; i < width; i += kGateThreads) {
    const int c = c0 + i;
    const float z = to_f32(zrow[c]);
    const float v = fmaf(Dskip[c / P], xrow[c], orow[c]) * (z * sigmoid_acc(z));
    y[(size_t)t * inner + c] = from_f32<T>(v * inv * w[c]);
  }
}

// The same, a warp a (token, slice) that holds it in registers, four neighbouring channels a lane at a time: slices of up to
// 128 VPL channels (a multiple of 4), P, the columns and the row strides multiples of 4, rows on 16 (bfloat16: 8) bytes.
// One pass over 201 MB for 2,048 tokens of 8,192 channels in 8 slices, no barrier: 97 us before, 66 with the accurate sigmoid and
// all rows at once, 54 so.
constexpr int kGateWarps = 8;
template <typename T, int VPL>
__global__ void __launch_bounds__(kGateWarps * 32, VPL == 8 ? 3 : 4)   // (loads under way count)
ssm_gate_norm_vec_kernel(T* __restrict__ y, const float* __restrict__ o, const float* __restrict__ xs,
                         const T* __restrict__ proj, int ld, int oz, const float* __restrict__ Dskip,
                         const float* __restrict__ w, int P, int inner, int parts, float eps, int units) {
  ccb::pdl_begin();
  const int unit = blockIdx.x * kGateWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (unit >= units) return;
  const int t = unit / parts, width = inner / parts, c0 = (unit - t * parts) * width;
  const float* orow = o + (size_t)t * inner + c0;
  const float* xrow = xs + (size_t)t * inner + c0;
  const T* zrow = proj + (size_t)t * ld + oz + c0;
  float4 v[VPL];
  typename In4<T>::Raw z[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = 4 * lane + 128 * i;
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    z[i] = {};
    if (c < width) {
      v[i] = *reinterpret_cast<const float4*>(orow + c);
      z[i] = *reinterpret_cast<const typename In4<T>::Raw*>(zrow + c);
    }
  }
#pragma unroll
  for (int i = 0; i < VPL; ++i) {   // (x goes in as it comes: three rows at once would leave an SM half its warps)
    const int c = 4 * lane + 128 * i;
    if (c >= width) continue;
    const float4 x = *reinterpret_cast<const float4*>(xrow + c);
    const float d = Dskip[(c0 + c) / P];
    v[i].x = fmaf(d, x.x, v[i].x);
    v[i].y = fmaf(d, x.y, v[i].y);
    v[i].z = fmaf(d, x.z, v[i].z);
    v[i].w = fmaf(d, x.w, v[i].w);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const float4 g = silu4_of<T>(In4<T>::value(z[i]));
    v[i].x *= g.x; v[i].y *= g.y; v[i].z *= g.z; v[i].w *= g.w;
    ss += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
  }
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss / (float)width + eps);
  T* yrow = y + (size_t)t * inner + c0;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = 4 * lane + 128 * i;
    if (c >= width) continue;
    const float4 ww = *reinterpret_cast<const float4*>(w + c0 + c);
    const float4 r = make_float4(v[i].x * inv * ww.x, v[i].y * inv * ww.y, v[i].z * inv * ww.z, v[i].w * inv * ww.w);
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(yrow + c) = r;
    } else {
      const __nv_bfloat162 a = __floats2bfloat162_rn(r.x, r.y), b = __floats2bfloat162_rn(r.z, r.w);
      *reinterpret_cast<uint2*>(yrow + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
  }
}

template <typename T>
bool launch_gate_norm_vec(void* y, const float* o, const float* xs, const void* proj, int ld, int oz, const float* Dskip,
                          const float* w, int rows, int H, int P, int parts, float eps, cudaStream_t stream) {
  const int inner = H * P, width = inner / parts;
  const auto bits = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  if (width % 4 || P % 4 || ld % 4 || oz % 4 || width > 1024 || (long long)rows * parts > 0x7fffffffll ||
      ((bits(o) | bits(xs) | bits(w)) & 15) || ((bits(y) | bits(proj)) % (4 * sizeof(T))))
    return false;
  const int units = rows * parts, blocks = (units + kGateWarps - 1) / kGateWarps;
#define CCB_GATE(VPL)                                                                                                   \
  ccb_launch(ssm_gate_norm_vec_kernel<T, VPL>, blocks, kGateWarps * 32, 0, stream, (T*)y, o, xs, (const T*)proj, ld, oz, \
             Dskip, w, P, inner, parts, eps, units)
  if (width <= 128) CCB_GATE(1);
  else if (width <= 256) CCB_GATE(2);
  else if (width <= 512) CCB_GATE(4);
  else CCB_GATE(8);
#undef CCB_GATE
  return true;
}

}  // namespace

CCB_API int ccb_ssm_prepare(const void* proj, int ld, int ox, int odt, const float* conv_w, const float* conv_b,
                            int taps, const void* conv_state, const float* A_log, const float* dt_bias,
                            const int* entry_of_token, const int* cu_q, const int* state_slot, float* xs, float* bs,
                            float* cs, float* dts, float* as, int rows, int H, int P, int G, int N, int shift_single,
                            int chunk_from, void* b_hi, void* b_lo, void* c_hi, void* c_lo, float* log_a, float* log_dt,
                            int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (H <= 0 || P <= 0 || G <= 0 || N <= 0 || H % G || taps < 1 || taps > 64) return CCB_REFUSE_SIZE;
  if (proj == nullptr || conv_w == nullptr || (taps > 1 && conv_state == nullptr)) return CCB_REFUSE_ARG;
  const int threads = 256;
  const int inner_ = H * P, gn_ = G * N;
  const bool vec = inner_ % 4 == 0 && gn_ % 4 == 0 && ox % 4 == 0 && ld % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(proj) | reinterpret_cast<uintptr_t>(conv_state) |
                     reinterpret_cast<uintptr_t>(conv_w) | reinterpret_cast<uintptr_t>(conv_b) |
                     reinterpret_cast<uintptr_t>(xs) | reinterpret_cast<uintptr_t>(bs) |
                     reinterpret_cast<uintptr_t>(cs)) & 15) == 0;
  // (rows for chunks: the caller asks for them with the sizes and addresses that the vector kernel takes)
  const SsmChunkRows chunk{chunk_from < 0 ? rows : chunk_from, (__nv_bfloat16*)b_hi, (__nv_bfloat16*)b_lo, (__nv_bfloat16*)c_hi,
                           (__nv_bfloat16*)c_lo, log_a, log_dt};
  if (chunk_from >= 0 && (!vec || !b_hi || !b_lo || !c_hi || !c_lo || !log_a || !log_dt ||
                          ((reinterpret_cast<uintptr_t>(b_hi) | reinterpret_cast<uintptr_t>(b_lo) |
                            reinterpret_cast<uintptr_t>(c_hi) | reinterpret_cast<uintptr_t>(c_lo)) & 7)))
    return CCB_REFUSE_ARG;
  if (vec && taps <= 4 && rows <= kSsmRun * 65535 && (long long)rows * ((inner_ + 2 * gn_) / 4 + H) >= kSsmRunUnits && (dtype == CCB_F32 || dtype == CCB_BF16)) {
    const dim3 grid(((inner_ + 2 * gn_) / 4 + H + threads - 1) / threads, (rows + kSsmRun - 1) / kSsmRun);
#define CCB_RUN(TT, TAPS)                                                                                                    \
  ccb_launch(ssm_prepare_run_kernel<TT, TAPS>, grid, threads, 0, stream, (const TT*)proj, ld, ox, odt, conv_w, conv_b,      \
             (const TT*)conv_state, A_log, dt_bias, entry_of_token, cu_q, state_slot, xs, bs, cs, dts, as, rows, H, P, G, N, \
             (TT*)conv_state, shift_single, chunk)
#define CCB_RUN_TAPS(TT)                \
  do {                                  \
    if (taps == 1) CCB_RUN(TT, 1);      \
    else if (taps == 2) CCB_RUN(TT, 2); \
    else if (taps == 3) CCB_RUN(TT, 3); \
    else CCB_RUN(TT, 4);                \
  } while (0)
    if (dtype == CCB_F32) CCB_RUN_TAPS(float);
    else CCB_RUN_TAPS(__nv_bfloat16);
#undef CCB_RUN_TAPS
#undef CCB_RUN
    return ccb_launch_status();
  }
  if (vec && (dtype == CCB_F32 || dtype == CCB_BF16)) {
    const size_t total4 = (size_t)rows * ((inner_ + 2 * gn_) / 4 + H);
    const size_t want4 = (total4 + threads - 1) / threads;
    const int blocks4 = (int)(want4 < 148 * 32 ? want4 : 148 * 32);
    if (dtype == CCB_F32)
      ccb_launch(ssm_prepare_vec_kernel<float>, blocks4, threads, 0, stream, (const float*)proj, ld, ox, odt, conv_w,
                 conv_b, taps, (const float*)conv_state, A_log, dt_bias, entry_of_token, cu_q, state_slot, xs, bs, cs,
                 dts, as, rows, H, P, G, N, (float*)conv_state, shift_single, chunk);
    else
      ccb_launch(ssm_prepare_vec_kernel<__nv_bfloat16>, blocks4, threads, 0, stream, (const __nv_bfloat16*)proj, ld, ox,
                 odt, conv_w, conv_b, taps, (const __nv_bfloat16*)conv_state, A_log, dt_bias, entry_of_token, cu_q,
                 state_slot, xs, bs, cs, dts, as, rows, H, P, G, N, (__nv_bfloat16*)conv_state, shift_single, chunk);
    return ccb_launch_status();
  }
  const size_t total = (size_t)rows * (H * P + 2 * G * N + H);
  const size_t want = (total + threads - 1) / threads;
  const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
  if (dtype == CCB_F32)
    ccb_launch(ssm_prepare_kernel<float>, blocks, threads, 0, stream, (const float*)proj, ld, ox, odt, conv_w, conv_b,
               taps, (const float*)conv_state, A_log, dt_bias, entry_of_token, cu_q, state_slot, xs, bs, cs, dts, as,
               rows, H, P, G, N, (float*)conv_state, shift_single);
  else if (dtype == CCB_BF16)
    ccb_launch(ssm_prepare_kernel<__nv_bfloat16>, blocks, threads, 0, stream, (const __nv_bfloat16*)proj, ld, ox, odt,
               conv_w, conv_b, taps, (const __nv_bfloat16*)conv_state, A_log, dt_bias, entry_of_token, cu_q,
               state_slot, xs, bs, cs, dts, as, rows, H, P, G, N, (__nv_bfloat16*)conv_state, shift_single);
  else
    return CCB_REFUSE_DTYPE;
  return ccb_launch_status();
}

CCB_API int ccb_conv_state_shift(const void* rows, int ld, int taps, int C, void* state, const int* cu_q,
                                 const int* state_slot, int entry0, int n_entries, int n_slots, int dtype,
                                 cudaStream_t stream) {
  if (n_entries <= 0 || taps <= 1) return 0;
  if (C <= 0) return CCB_REFUSE_SIZE;
  const size_t total = (size_t)n_entries * C;
  const int threads = 256;
  const size_t want = (total + threads - 1) / threads;
  const int blocks = (int)(want < 148 * 16 ? want : 148 * 16);
  if (dtype == CCB_F32)
    ccb_launch(conv_state_shift_kernel<float>, blocks, threads, 0, stream, (const float*)rows, ld, taps, C,
               (float*)state, cu_q, state_slot, entry0, n_entries, n_slots);
  else if (dtype == CCB_BF16)
    ccb_launch(conv_state_shift_kernel<__nv_bfloat16>, blocks, threads, 0, stream, (const __nv_bfloat16*)rows, ld, taps,
               C, (__nv_bfloat16*)state, cu_q, state_slot, entry0, n_entries, n_slots);
  else
    return CCB_REFUSE_DTYPE;
  return ccb_launch_status();
}

CCB_API int ccb_ssm_gate_norm(void* y, const float* o, const float* xs, const void* proj, int ld, int oz,
                              const float* Dskip, const float* w, int rows, int H, int P, int parts, float eps,
                              int dtype, cudaStream_t stream) {
  if (rows <= 0) return 0;
  const int inner = H * P;
  if (H <= 0 || P <= 0 || parts <= 0 || inner % parts) return CCB_REFUSE_SIZE;
  // A warp a slice from 1,024 slices on; a block each while there are few (8 slices a token, block / warp: 16 tokens 21.3 /
  // 22.7 us, 64 tokens 22.4 / 22.6, 128 tokens 24.6 / 24.0, 512 tokens 43.7 / 35.2)
  if ((long long)rows * parts >= 1024 &&
      ((dtype == CCB_F32 && launch_gate_norm_vec<float>(y, o, xs, proj, ld, oz, Dskip, w, rows, H, P, parts, eps, stream)) ||
       (dtype == CCB_BF16 && launch_gate_norm_vec<__nv_bfloat16>(y, o, xs, proj, ld, oz, Dskip, w, rows, H, P, parts, eps, stream))))
    return ccb_launch_status();
  dim3 grid(rows, parts);   // (slices or addresses that the vector form does not take)
  if (dtype == CCB_F32)
    ccb_launch(ssm_gate_norm_kernel<float>, grid, dim3(kGateThreads), 0, stream, (float*)y, o, xs, (const float*)proj,
               ld, oz, Dskip, w, P, inner, parts, eps);
  else if (dtype == CCB_BF16)
    ccb_launch(ssm_gate_norm_kernel<__nv_bfloat16>, grid, dim3(kGateThreads), 0, stream, (__nv_bfloat16*)y, o, xs,
               (const __nv_bfloat16*)proj, ld, oz, Dskip, w, P, inner, parts, eps);
  else
    return CCB_REFUSE_DTYPE;
  return ccb_launch_status();
}
