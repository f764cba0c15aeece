// The gated recurrences of csrc/delta_rule.cu over portions of prompts, in chunks of 64 tokens on tensor cores:
//
//   S <- diag(g_t) S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t        (delta rule)
//   S <- diag(g_t) S + k_t v_t^T;                     o_t = S^T q_t                              (without: u = v)
//
// with one decay per key channel or one per head.  With c_t the sum of log g over the chunk up to t (per channel), S0
// the memory before the chunk and x . y over key channels,
//
//   M_ts = (k_t e^{c_t - c_s}) . k_s,   P_ts = (q_t e^{c_t - c_s}) . k_s
//   (I + strictly_lower(diag(beta) M)) [W | U] = diag(beta) [K e^c | V]
//   u = U - W S0;   o = (Q e^c) S0 + lower(P) u;   S = e^{c_64} S0 + (K e^{c_64 - c})^T u
//
// so only the last line walks the chunks in order; everything before it is independent of the memory.  Two kernels:
//
//   chunk_prepare  a block per (chunk, head): the sums of logarithms, M and P, the scaled rows of q and k, and the
//                  triangular solve: the four 16 x 16 blocks on the diagonal are inverted in float, the rest are products
//                  of a warp's 32 columns, transposed, so that one block's result is the next one's operand as it is
//   chunk_walk     a block per (request, head, 32 value columns), eight warps: the memory in float registers, four
//                  products a chunk on mma.sync; a warp takes 16 rows x 16 columns of u and o and 16 key channels of S
//
// Exponents of decays are never positive between runs of 16 tokens, where both factors refer to a place between them.
// Within a run they refer to its eighth token where every channel stays within 2^-55 of it, which slow and ordinary
// decays do; else every pair's decay is taken per channel as it is, one exponential each.  Logarithms are summed within a run and runs are added up, so
// that a difference never cancels more than a run's sum.  What the model computes in 32 bits stays so to about 2^-17:
// logarithms, sums, exponentials, the solve and the memory are float, and every operand of a product (rows, scores,
// memory) goes in as TWO bfloat16, its rounding and what the rounding left, in three products.  A decay below 2^-115
// counts as that: it keeps nothing that a float can tell from zero.
// A number that is not finite must not reach the tokens before it, whose share of it is a zero that would still be
// multiplied by it: among the operands whose sum runs over tokens (the solve's right sides, u) it enters as zero, and what
// it belongs to, from its token on, is made NaN afterwards.
//
// Bound by: the walk by the chain of its products (one block of eight warps an SM, an instruction on 0.30 of the cycles),
// the preparation by what it issues (0.5).  Measured on B200, 2,048 tokens of one request, 32 heads of 128 x 128 with a
// decay per channel and the delta rule: 163 + 95 us (with what it reads loaded as it is needed 199, with the solve's operands split
// again by every 16 columns 8 more); token by token 959 us.  Outputs and memory are right to 5e-6 in the
// 2-norm, token by token to 1e-7 to 4e-7; in a layer's results, whose rows are bfloat16 (3.7e-3), neither shows.
#include "common.cuh"
#include "mma_common.cuh"
#include <math_constants.h>
#include <type_traits>

using namespace ccb;

namespace {

constexpr int kChunk = 64;
constexpr int kThreads = 256;
constexpr int kRun = 16;           // tokens of a run
constexpr float kLeastLog2 = -115.f;
constexpr float kSteepLog2 = 55.f;   // (2^110 times 128 products stays in a float, also in places that nobody sees)

// Gated linear attention's rows as the projections left them, in place of q, k, v and g: q times q_mult, k and v; the decay is
// sigmoid(a + bias)^(1 / tau).  Measured on B200, 1,537 tokens of three requests, 16 heads of 128, a layer: 173 -> 162 us (the rows'
// kernel of 18 us gone, preparation 33 -> 40, walk 40 -> 43).
// The delta rule takes only its decays so, exp(-exp(A_log) softplus(a + bias)): at 2,048 tokens of 32 heads the rows' kernel 87 -> 72 us,
// the preparation 7 more (a layer 605 -> 596, both with a faster activation in the rows' kernel).  Its q, k and v too, convolved by the preparation: 270 without a rows' kernel, 617.
struct RawRows {
  const __nv_bfloat16 *q, *k, *v, *a;   // q, k [T, ld] with head h at column h DK, v [T, ld] at h dv, a [T, lda] at h DK
  int ld, lda;
  const float* bias;                    // [H DK] or null
  float q_mult, inv_tau;
  const float* A_log;                   // [H] (delta rule)
};

struct ChunkRows {
  const float *q, *k, *v, *g, *beta;   // q, k [T, G, DK]; v [T, H, dv]; g [T, H, DK], or [T, H] with one decay a head
  __nv_bfloat16 *qs, *ks, *w;          // [T, H, 2, DK]: a row's bfloat16 values, then what their rounding left
  float* u;                            // [T, H, dv]
  __nv_bfloat16* p;                    // [T, H, 2, 64]
  float* keep;                         // [T / 64 + entries, H, DK]: e^{c_64} of a chunk
  float *state, *out;                  // [slots, H, dv, DK], [T, H, dv]
  const int *cu_q, *state_slot;
  int entry0, G, H, dv, n_slots;
  RawRows raw;
};

__device__ __forceinline__ float4 four(const __nv_bfloat16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ void copy16(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }   // (this thread's)

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// bfloat16 pair of (x, y) and of what their rounding left
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 f = __bfloat1622float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_bf16(x - f.x, y - f.y);
}

// c += a b with both operands as two bfloat16
__device__ __forceinline__ void mma3(float* c, const uint32_t* ah, const uint32_t* al, uint32_t bh0, uint32_t bh1, uint32_t bl0,
                                     uint32_t bl1) {
  mma_bf16_16816(c, al, bh0, bh1);
  mma_bf16_16816(c, ah, bl0, bl1);
  mma_bf16_16816(c, ah, bh0, bh1);
}

// rows of DK floats: the eight-float groups of neighbouring rows sit in different banks
template <int DK> __device__ __forceinline__ int at(int row, int col) { return row * DK + (col ^ ((row & 3) << 3)); }

constexpr int kPitchL = kChunk;
__device__ __forceinline__ int lat(int t, int s) { return t * kPitchL + (s ^ ((t & 3) << 3)); }   // place (t, s) of l_s

template <int DK, bool DELTA, bool HEAD> struct PrepShape {
  static constexpr int kC = HEAD ? kChunk : kChunk * DK;   // sums of logarithms
  static constexpr int kFloats = 2 * kChunk * DK + kC + (DELTA ? kChunk * kPitchL : 0) + kChunk;   // (two blocks an SM)
  static constexpr int kBytes = kFloats * 4 + 48;
};

// 32 values a lane, one for each lane: the sum of value i over all lanes ends in lane i
__device__ __forceinline__ float transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float mine = up ? v[i + o] : v[i], other = up ? v[i] : v[i + o];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
    }
  }
  return v[0];
}

// A lane's eight right sides of a run (two columns, four tokens each, as the solve holds them) with those that are not finite
// as zeros, and by column the first token that has one (kRun: none).  A call of its own: unrolled into the solve, code
// that hardly ever runs made the preparation of 2,048 tokens of 32 heads 201 us by its length, 193 so (187 without any).
struct RunSides {
  float x[8];
  int bad[2];
};
__device__ __noinline__ RunSides separate(float x0, float x1, float x2, float x3, float x4, float x5, float x6, float x7) {
  const int tig = threadIdx.x & 3;
  RunSides r{{x0, x1, x2, x3, x4, x5, x6, x7}, {kRun, kRun}};
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (!is_finite(r.x[i])) {
      r.bad[(i >> 1) & 1] = min(r.bad[(i >> 1) & 1], (i >> 2) * 8 + 2 * tig + (i & 1));
      r.x[i] = 0.f;
    }
#pragma unroll
  for (int up = 0; up < 2; ++up) {   // (the four lanes of a column)
    r.bad[up] = min(r.bad[up], __shfl_xor_sync(0xffffffffu, r.bad[up], 1));
    r.bad[up] = min(r.bad[up], __shfl_xor_sync(0xffffffffu, r.bad[up], 2));
  }
  return r;
}

template <int DK, bool DELTA, bool HEAD, bool RAW = false>
__global__ void __launch_bounds__(kThreads, 2)
chunk_prepare_kernel(const ChunkRows a) {
  ccb::pdl_begin();
  using Sh = PrepShape<DK, DELTA, HEAD>;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;                         // [64][DK]
  float* k_s = q_s + kChunk * DK;
  float* c_s = k_s + kChunk * DK;            // [64][DK] or [64]: log2 of the decay since the token's run began
  float* l_s = c_s + Sh::kC;                 // [64][64]: diag(beta) M below the diagonal
  float* b_s = l_s + (DELTA ? kChunk * kPitchL : 0);
  int* next_item = reinterpret_cast<int*>(b_s + kChunk);
  int* steep = next_item + 1;                // [8 warps]: a bit for each run that takes every pair's decay by itself

  const int e = a.entry0 + blockIdx.z, h = blockIdx.y, chunk = blockIdx.x;
  const int first = a.cu_q[e], n = a.cu_q[e + 1] - first;
  const int slot = a.state_slot[e];
  if (slot < 0 || slot >= a.n_slots || chunk * kChunk >= n) return;
  const int r0 = first + chunk * kChunk, cnt = min(kChunk, n - chunk * kChunk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kvh = h / (a.H / a.G);

  // Float rows go straight to shared memory while the logarithms below are loaded and taken.  (Through registers, with a barrier
  // before the logarithms: 174 us, 163 so; the logarithms' loads before the rows': 185.)
  for (int i = tid; i < kChunk * DK / 4; i += kThreads) {
    const int t = i / (DK / 4), c = 4 * (i % (DK / 4));
    float* q_at = q_s + at<DK>(t, c);
    float* k_at = k_s + at<DK>(t, c);
    if (t >= cnt) {
      *reinterpret_cast<float4*>(q_at) = *reinterpret_cast<float4*>(k_at) = make_float4(0.f, 0.f, 0.f, 0.f);
    } else if (RAW && !DELTA) {
      const size_t row = (size_t)(r0 + t) * a.raw.ld + kvh * DK + c;
      const float4 q = four(a.raw.q + row);
      *reinterpret_cast<float4*>(k_at) = four(a.raw.k + row);
      *reinterpret_cast<float4*>(q_at) = make_float4(q.x * a.raw.q_mult, q.y * a.raw.q_mult, q.z * a.raw.q_mult, q.w * a.raw.q_mult);
    } else {
      const size_t row = ((size_t)(r0 + t) * a.G + kvh) * DK + c;
      copy16(q_at, a.q + row);
      copy16(k_at, a.k + row);
    }
  }
  if (tid < kChunk) b_s[tid] = DELTA && tid < cnt ? a.beta[(size_t)(r0 + tid) * a.H + h] : 0.f;
  if (tid == 0) *next_item = 0;
  auto log_decay = [](float g) {
    const float x = log2f(g);
    return x < kLeastLog2 ? kLeastLog2 : x;
  };
  if constexpr (HEAD) {
    if (warp == 0) {   // two tokens a lane, eight lanes a run
      float x[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = 2 * lane + i;
        x[i] = t < cnt ? log_decay(a.g[(size_t)(r0 + t) * a.H + h]) : 0.f;
      }
      float before = x[0] + x[1];
#pragma unroll
      for (int o = 1; o < kRun / 2; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, before, o, kRun / 2);
        if ((lane & (kRun / 2 - 1)) >= o) before += y;
      }
      before = __shfl_up_sync(0xffffffffu, before, 1, kRun / 2);
      if ((lane & (kRun / 2 - 1)) == 0) before = 0.f;
      c_s[2 * lane] = before + x[0];
      c_s[2 * lane + 1] = before + x[0] + x[1];
    }
  } else {   // a thread a channel and some runs
    constexpr int PT = kChunk * DK / kThreads;
    static_assert(PT % kRun == 0, "whole runs");
    const int d = tid % DK, part = tid / DK;
    float x[PT];
#pragma unroll
    for (int i = 0; i < PT; ++i) {
      const int t = part * PT + i;
      if (RAW) x[i] = t < cnt ? __bfloat162float(a.raw.a[(size_t)(r0 + t) * a.raw.lda + h * DK + d]) : 0.f;
      else x[i] = t < cnt ? a.g[((size_t)(r0 + t) * a.H + h) * DK + d] : 1.f;
    }
    const float bias = RAW && a.raw.bias != nullptr ? a.raw.bias[h * DK + d] : 0.f;
    // (straight from the projections' row: a decay near one would lose its logarithm's places to its own rounding)
    const float rate = RAW && DELTA ? expf(a.raw.A_log[h]) : 0.f;
    auto log_raw = [&](float z) {
      float l;
      if (DELTA) l = -rate * (z > 20.f ? z : log1pf(expf(z))) * 1.44269504088896f;
      else l = (fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * (a.raw.inv_tau * 1.44269504088896f);
      return l < kLeastLog2 ? kLeastLog2 : l;
    };
    int mine = 0;
#pragma unroll
    for (int m = 0; m < PT / kRun; ++m) {
      float sum = 0.f, first_sum = 0.f, mid = 0.f;
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        if (RAW) sum += part * PT + m * kRun + i < cnt ? log_raw(x[m * kRun + i] + bias) : 0.f;
        else sum += log_decay(x[m * kRun + i]);
        c_s[at<DK>(part * PT + m * kRun + i, d)] = sum;
        if (i == 0) first_sum = sum;
        if (i == kRun / 2 - 1) mid = sum;
      }
      if (!(first_sum - mid <= kSteepLog2 && mid - sum <= kSteepLog2)) mine |= 1 << (part * (PT / kRun) + m);
    }
    mine = __reduce_or_sync(0xffffffffu, mine);
    if (lane == 0) steep[warp] = mine;
  }
  copies_landed();
  __syncthreads();
  auto in_run = [&](int t, int d) { return HEAD ? c_s[t] : c_s[at<DK>(t, d)]; };
  // the decay of whole runs lo .. hi - 1
  auto over_runs = [&](int lo, int hi, int d) {
    float sum = 0.f;
#pragma unroll
    for (int m = 0; m < kChunk / kRun; ++m)
      if (m >= lo && m < hi) sum += in_run(m * kRun + kRun - 1, d);
    return sum;
  };
  const size_t p_row = (size_t)a.H * 2 * kChunk;   // elements from a token's scores to the next one's
  __nv_bfloat16* p_out = a.p + ((size_t)r0 * a.H + h) * 2 * kChunk;

  // ---- blocks of 16 x 16 pairs, a warp each, to whoever is free: rows of run i, columns of run j
  const int gid = lane >> 2, tig = lane & 3;
  int steep_runs = 0;
  if (!HEAD)
    for (int w = 0; w < kThreads / 32; ++w) steep_runs |= steep[w];
  auto take = [&]() {
    int item = 0;
    if (lane == 0) item = atomicAdd(next_item, 1);
    return __shfl_sync(0xffffffffu, item, 0);
  };
  constexpr int kPairs = 10;
  int item = take();
  for (; item < kPairs; item = take()) {
    int i = 0, j = item;
    while (j > i) j -= ++i;
    if (i * kRun >= cnt || (i == j && (steep_runs >> i & 1))) continue;
    // the place that both factors refer to: the end of run j, or the middle of a run
    const int edge = (j + 1) * kRun - 1 - (i == j ? kRun / 2 : 0);
    float sq[2][4], sk[2][4];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) sq[x][y] = sk[x][y] = 0.f;
#pragma unroll 2
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t qh[4], ql[4], kh[4], kl[4], bh[2][2], bl[2][2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int col = ks * 16 + 2 * tig + 8 * half;
        float2 ce = make_float2(0.f, 0.f), mid = ce;   // of run j, and of the runs between j and i
        if (!HEAD) {
          ce = *reinterpret_cast<const float2*>(c_s + at<DK>(edge, col));
          for (int m = j + 1; m < i; ++m) {
            const float2 c = *reinterpret_cast<const float2*>(c_s + at<DK>(m * kRun + kRun - 1, col));
            mid.x += c.x;
            mid.y += c.y;
          }
        }
#pragma unroll
        for (int up = 0; up < 2; ++up) {
          const int t = i * kRun + gid + 8 * up;
          float2 q = *reinterpret_cast<const float2*>(q_s + at<DK>(t, col));
          float2 k = make_float2(0.f, 0.f);
          if (DELTA) k = *reinterpret_cast<const float2*>(k_s + at<DK>(t, col));
          if (!HEAD) {
            const float2 c = *reinterpret_cast<const float2*>(c_s + at<DK>(t, col));
            if (i == j) mid = make_float2(-ce.x, -ce.y);
            const float fx = ex2(c.x + mid.x), fy = ex2(c.y + mid.y);
            q.x *= fx; q.y *= fy;
            k.x *= fx; k.y *= fy;
          }
          split2(q.x, q.y, qh[2 * half + up], ql[2 * half + up]);
          if (DELTA) split2(k.x, k.y, kh[2 * half + up], kl[2 * half + up]);
        }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          const int s = j * kRun + nb * 8 + gid;
          float2 k = *reinterpret_cast<const float2*>(k_s + at<DK>(s, col));
          if (!HEAD) {
            const float2 c = *reinterpret_cast<const float2*>(c_s + at<DK>(s, col));
            k.x *= ex2(ce.x - c.x);
            k.y *= ex2(ce.y - c.y);
          }
          split2(k.x, k.y, bh[nb][half], bl[nb][half]);
        }
      }
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        mma3(sq[nb], qh, ql, bh[nb][0], bh[nb][1], bl[nb][0], bl[nb][1]);
        if (DELTA) mma3(sk[nb], kh, kl, bh[nb][0], bh[nb][1], bl[nb][0], bl[nb][1]);
      }
    }
#pragma unroll
    for (int nb = 0; nb < 2; ++nb)
#pragma unroll
      for (int up = 0; up < 2; ++up) {
        const int t = i * kRun + gid + 8 * up, s = j * kRun + nb * 8 + 2 * tig;
        float f[2] = {1.f, 1.f};
        if (HEAD) {
          const int end = (j + 1) * kRun - 1;
#pragma unroll
          for (int x = 0; x < 2; ++x)
            f[x] = ex2(i == j ? fminf(c_s[t] - c_s[s + x], 0.f) : c_s[t] + (over_runs(j + 1, i, 0) + (c_s[end] - c_s[s + x])));
        }
        const float p0 = s <= t ? sq[nb][2 * up] * f[0] : 0.f, p1 = s + 1 <= t ? sq[nb][2 * up + 1] * f[1] : 0.f;
        if (t < cnt) {
          uint32_t hi, lo;
          split2(p0, p1, hi, lo);
          *reinterpret_cast<uint32_t*>(p_out + t * p_row + s) = hi;
          *reinterpret_cast<uint32_t*>(p_out + t * p_row + kChunk + s) = lo;
        }
        if (DELTA) {
          const float b = b_s[t];
          l_s[lat(t, s)] = s < t ? sk[nb][2 * up] * f[0] * b : 0.f;
          l_s[lat(t, s + 1)] = s + 1 < t ? sk[nb][2 * up + 1] * f[1] * b : 0.f;
        }
      }
  }
  // ---- pairs within a run, a decay for every pair and channel: a warp a row, its lanes the channels.  Rows with many
  // pairs first.
  if (!HEAD && steep_runs) {
    constexpr int CL = DK / 32;   // channels a lane
    for (; item < kPairs + kChunk; item = take()) {
      const int run = (item - kPairs) & 3, lt = kRun - 1 - ((item - kPairs) >> 2), t = run * kRun + lt;
      if (t >= cnt || !(steep_runs >> run & 1)) continue;
      float q[CL], k[CL], c[CL], v[32];
#pragma unroll
      for (int x = 0; x < CL; ++x) {
        q[x] = q_s[at<DK>(t, lane + 32 * x)];
        k[x] = k_s[at<DK>(t, lane + 32 * x)];
        c[x] = c_s[at<DK>(t, lane + 32 * x)];
      }
#pragma unroll
      for (int s = 0; s < kRun; ++s) {
        v[s] = v[kRun + s] = 0.f;
        if (s > lt) continue;
        const int row = run * kRun + s;
#pragma unroll
        for (int x = 0; x < CL; ++x) {
          const float ke = k_s[at<DK>(row, lane + 32 * x)] * ex2(c[x] - c_s[at<DK>(row, lane + 32 * x)]);
          v[s] = fmaf(q[x], ke, v[s]);
          if (DELTA) v[kRun + s] = fmaf(k[x], ke, v[kRun + s]);
        }
      }
      const float sum = transpose_sum(v, lane);
      const int s = lane & 15;
      if (lane < kRun) {
        const float x = s <= lt ? sum : 0.f;
        const __nv_bfloat16 hi = __float2bfloat16_rn(x);
        p_out[t * p_row + run * kRun + s] = hi;
        p_out[t * p_row + kChunk + run * kRun + s] = __float2bfloat16_rn(x - __bfloat162float(hi));
      } else if (DELTA) {
        l_s[lat(t, run * kRun + s)] = s < lt ? sum * b_s[t] : 0.f;
      }
    }
  }
  // ---- the rows that meet the memory: q e^c, k e^{c_64 - c}, and e^{c_64}
  {   // a thread two channels of some rows of a run
    constexpr int PARTS = kThreads / (DK / 2), ROWS = kChunk / PARTS;
    const int d = 2 * (tid % (DK / 2)), t0 = (tid / (DK / 2)) * ROWS, run = t0 / kRun;
    const float before[2] = {over_runs(0, run, d), over_runs(0, run, d + 1)};
    const float after[2] = {over_runs(run + 1, kChunk / kRun, d), over_runs(run + 1, kChunk / kRun, d + 1)};
    const float end[2] = {in_run(run * kRun + kRun - 1, d), in_run(run * kRun + kRun - 1, d + 1)};   // (rows past the end decay nothing)
#pragma unroll 4
    for (int t = t0; t < min(t0 + ROWS, cnt); ++t) {
      const float2 q = *reinterpret_cast<const float2*>(q_s + at<DK>(t, d)), k = *reinterpret_cast<const float2*>(k_s + at<DK>(t, d));
      const float c0 = in_run(t, d), c1 = in_run(t, d + 1);
      const size_t row = ((size_t)(r0 + t) * a.H + h) * 2 * DK + d;
      uint32_t hi, lo;
      split2(q.x * ex2(before[0] + c0), q.y * ex2(before[1] + c1), hi, lo);
      *reinterpret_cast<uint32_t*>(a.qs + row) = hi;
      *reinterpret_cast<uint32_t*>(a.qs + row + DK) = lo;
      split2(k.x * ex2(after[0] + (end[0] - c0)), k.y * ex2(after[1] + (end[1] - c1)), hi, lo);
      *reinterpret_cast<uint32_t*>(a.ks + row) = hi;
      *reinterpret_cast<uint32_t*>(a.ks + row + DK) = lo;
    }
  }
  const int place = (first >> 6) + e + chunk;   // (distinct: an entry's last chunk comes before the next entry's first)
  for (int d = tid; d < DK; d += kThreads) a.keep[((size_t)place * a.H + h) * DK + d] = ex2(over_runs(0, kChunk / kRun, d));

  // ---- the triangular solve for X = [W | U]: with L the strictly lower blocks, X_i = (I + L_ii)^-1 (B_i - sum L_ij X_j)
  if constexpr (DELTA) {
    __syncthreads();
    // The values go where the queries were while the diagonal's blocks are inverted (values of more channels: read one by one).
    // Loaded where the solve needs them, each 16 x 16 block waited: 199 us, 174 so.
    const bool values_in = a.dv <= DK;
    if (values_in)
      for (int x = tid; x < cnt * (a.dv / 4); x += kThreads) {
        const int t = x / (a.dv / 4), c = 4 * (x - t * (a.dv / 4));
        copy16(q_s + at<DK>(t, c), a.v + ((size_t)(r0 + t) * a.H + h) * a.dv + c);
      }
    // (as operands, two neighbouring columns as their two bfloat16 in the place of two floats: every 16 columns of X read them)
    if (tid < kChunk) {   // a thread a column of an inverse, which takes its block's place
      const int run = tid / kRun, c = tid % kRun;
      float y[kRun];
#pragma unroll
      for (int t = 0; t < kRun; ++t) {
        float x = t == c ? 1.f : 0.f;
        if (run * kRun + t < cnt) {
#pragma unroll
          for (int s = 0; s < t; ++s) x = fmaf(-l_s[lat(run * kRun + t, run * kRun + s)], y[s], x);
        }
        y[t] = x;
      }
      __syncwarp();
#pragma unroll
      for (int t = 0; t < kRun; ++t) {
        const float right = __shfl_xor_sync(0xffffffffu, y[t], 1);
        uint2 both;
        split2(y[t], right, both.x, both.y);
        if ((c & 1) == 0) *reinterpret_cast<uint2*>(l_s + lat(run * kRun + t, run * kRun + c)) = both;
      }
    } else {   // the blocks below them, negated
      constexpr int kRest = kThreads - kChunk;
      for (int x = tid - kChunk; x < 6 * kRun * kRun / 2; x += kRest) {
        const int b = x / (kRun * kRun / 2), i = b < 1 ? 1 : b < 3 ? 2 : 3, j = b - i * (i - 1) / 2;
        const int t = i * kRun + x % (kRun * kRun / 2) / (kRun / 2), s = j * kRun + 2 * (x % (kRun / 2));
        float* at = l_s + lat(t, s);
        const float2 l = *reinterpret_cast<const float2*>(at);
        uint2 both;
        split2(t < cnt ? -l.x : 0.f, t < cnt ? -l.y : 0.f, both.x, both.y);
        *reinterpret_cast<uint2*>(at) = both;
      }
    }
    copies_landed();
    __syncthreads();
    const int runs = (cnt + kRun - 1) / kRun;
    // A warp 16 columns at a time: the transposed block [columns, tokens] is an accumulator, and split in two an A operand
    for (int c0 = 16 * warp; c0 < DK + a.dv; c0 += 16 * (kThreads / 32)) {
      const bool is_w = c0 < DK;
      uint32_t xh[3][4], xl[3][4];   // X_j of the runs before
      float before[2] = {0.f, 0.f};
#pragma unroll
      for (int i = 0; i < kChunk / kRun; ++i) {
        if (i >= runs) break;
        float x[2][4];   // [8 tokens][place]
#pragma unroll
          for (int up = 0; up < 2; ++up) {
            const int col = c0 + gid + 8 * up;
#pragma unroll
            for (int nb = 0; nb < 2; ++nb)
#pragma unroll
              for (int y = 0; y < 2; ++y) {
                const int t = i * kRun + nb * 8 + 2 * tig + y;
                float b = 0.f;
                if (t < cnt)
                  b = is_w ? k_s[at<DK>(t, col)] * ex2(before[up] + in_run(t, col))
                           : values_in ? q_s[at<DK>(t, col - DK)] : a.v[((size_t)(r0 + t) * a.H + h) * a.dv + col - DK];
                x[nb][2 * up + y] = b * b_s[t];
              }
            if (is_w) before[up] += in_run(i * kRun + kRun - 1, col);
          }
#pragma unroll
        for (int j = 0; j < i; ++j) {
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) {
            uint32_t bh[2], bl[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int t = i * kRun + nb * 8 + gid;
              const uint2 l = *reinterpret_cast<const uint2*>(l_s + lat(t, j * kRun + 8 * half + 2 * tig));
              bh[half] = l.x;
              bl[half] = l.y;
            }
            mma3(x[nb], xh[j], xl[j], bh[0], bh[1], bl[0], bl[1]);
          }
        }
        int bad[2] = {kRun, kRun};   // by column: the first token of the run with no finite right side
        float most = 0.f;
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) most = largest(largest(most, x[nb][0], x[nb][1]), x[nb][2], x[nb][3]);
        const bool any_bad = __any_sync(0xffffffffu, !is_finite(most));
        if (any_bad) {
          const RunSides r = separate(x[0][0], x[0][1], x[0][2], x[0][3], x[1][0], x[1][1], x[1][2], x[1][3]);
#pragma unroll
          for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int y = 0; y < 4; ++y) x[nb][y] = r.x[4 * nb + y];
          bad[0] = r.bad[0];
          bad[1] = r.bad[1];
        }
        uint32_t ah[4], al[4];
#pragma unroll
          for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int up = 0; up < 2; ++up) {
              split2(x[nb][2 * up], x[nb][2 * up + 1], ah[2 * nb + up], al[2 * nb + up]);
              x[nb][2 * up] = x[nb][2 * up + 1] = 0.f;
            }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          uint32_t bh[2], bl[2];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const uint2 l = *reinterpret_cast<const uint2*>(l_s + lat(i * kRun + nb * 8 + gid, i * kRun + 8 * half + 2 * tig));
            bh[half] = l.x;
            bl[half] = l.y;
          }
          mma3(x[nb], ah, al, bh[0], bh[1], bl[0], bl[1]);
        }
        if (any_bad) {
#pragma unroll
          for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int y = 0; y < 4; ++y)
              if (nb * 8 + 2 * tig + (y & 1) >= bad[y >> 1]) x[nb][y] = CUDART_NAN_F;
        }
#pragma unroll
          for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int up = 0; up < 2; ++up) {
              uint32_t hi, lo;
              split2(x[nb][2 * up], x[nb][2 * up + 1], hi, lo);
              if (i < 3) {
                xh[i < 3 ? i : 0][2 * nb + up] = hi;
                xl[i < 3 ? i : 0][2 * nb + up] = lo;
              }
              const int col = c0 + gid + 8 * up;
#pragma unroll
              for (int y = 0; y < 2; ++y) {
                const int t = i * kRun + nb * 8 + 2 * tig + y;
                if (t >= cnt) continue;
                if (is_w) {
                  unsigned short* w = reinterpret_cast<unsigned short*>(a.w) + ((size_t)(r0 + t) * a.H + h) * 2 * DK + col;
                  w[0] = (unsigned short)(hi >> (16 * y));
                  w[DK] = (unsigned short)(lo >> (16 * y));
                } else {
                  a.u[((size_t)(r0 + t) * a.H + h) * a.dv + col - DK] = x[nb][2 * up + y];
                }
              }
            }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
constexpr int kCols = 32;          // value columns a block
constexpr int kPitch = kCols + 8;  // elements: eight rows of an ldmatrix fall into different banks

template <int DK, bool DELTA> struct WalkShape {
  static constexpr int kTile = 2 * kChunk * DK;                 // elements of the two halves of 64 rows
  static constexpr int kElements = (DELTA ? 3 : 2) * kTile + 2 * kChunk * kChunk + 2 * DK * kPitch + 2 * kChunk * kPitch;
  static constexpr int kBytes = kElements * 2;
};

template <int DK, bool DELTA, bool RAW = false>
__global__ void __launch_bounds__(kThreads)
chunk_walk_kernel(const ChunkRows a) {
  ccb::pdl_begin();
  using Sh = WalkShape<DK, DELTA>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(smem_raw);   // [2][64][DK], swizzled
  __nv_bfloat16* k_s = q_s + Sh::kTile;
  __nv_bfloat16* w_s = k_s + Sh::kTile;
  __nv_bfloat16* p_s = w_s + (DELTA ? Sh::kTile : 0);                // [2][64][64], swizzled
  __nv_bfloat16* s_hi = p_s + 2 * kChunk * kChunk;                   // [DK][kPitch]
  __nv_bfloat16* s_lo = s_hi + DK * kPitch;
  __nv_bfloat16* u_hi = s_lo + DK * kPitch;                          // [64][kPitch]
  __nv_bfloat16* u_lo = u_hi + kChunk * kPitch;

  // by column of the slice: the first token of a chunk whose u is not finite (64: none); and whether there is one
  __shared__ int bad_col[kCols], bad_any;
  const int e = a.entry0 + blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * kCols;
  const int slot = a.state_slot[e];
  const int r0 = a.cu_q[e], n = a.cu_q[e + 1] - r0;
  if (slot < 0 || slot >= a.n_slots || n <= 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  // 16 rows of the chunk, 16 columns of the slice.  Later rows meet more tokens, and the two warps of a scheduler share that (107 ->
  // 103.5 us; without the delta rule, where the update of S is all that follows, 43.0 / 43.4)
  const int wc = warp >> 2, wr = DELTA && wc == 1 ? 3 - (warp & 3) : warp & 3;

  // 64 rows of two halves of `COLS` elements each, a row (r0 + t, h), into two swizzled tiles
  auto issue = [&](__nv_bfloat16* dst, const __nv_bfloat16* src, int chunk, auto cols) {
    constexpr int COLS = decltype(cols)::value;
    const int t0 = chunk * kChunk;
#pragma unroll
    for (int i = 0; i < 2 * kChunk * (COLS / 8) / kThreads; ++i) {
      const int idx = tid + kThreads * i;
      const int row = idx / (COLS / 4), c = idx % (COLS / 4), half = c / (COLS / 8), c8 = c % (COLS / 8);
      const bool ok = t0 + row < n;
      cp_async16(smem_u32(dst + half * kChunk * COLS + swz<COLS>(row, c8)),
                 src + ((size_t)(r0 + t0 + (ok ? row : 0)) * a.H + h) * 2 * COLS + c * 8, ok);
    }
  };
  using Dk = std::integral_constant<int, DK>;
  using P64 = std::integral_constant<int, kChunk>;
  auto issue_read = [&](int chunk) {    // what meets the memory
    issue(q_s, a.qs, chunk, Dk{});
    if (DELTA) issue(w_s, a.w, chunk, Dk{});
    cp_async_commit();
  };
  auto issue_write = [&](int chunk) {   // what meets u
    issue(p_s, a.p, chunk, P64{});
    issue(k_s, a.ks, chunk, Dk{});
    cp_async_commit();
  };
  issue_read(0);
  if (tid < kCols) bad_col[tid] = kChunk;   // (read and written behind the barriers of a chunk)
  if (tid == 0) bad_any = 0;

  // S: key channels 16 warp .. + 15 (with 64 channels only the first four warps have some), all columns of the slice
  constexpr int SW = DK / 16;   // warps with channels
  float S[4][4];
  float* sp = a.state + ((size_t)slot * a.H + h) * (size_t)a.dv * DK;
  auto store_s = [&]() {
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
      for (int up = 0; up < 2; ++up) {
        const int row = warp * 16 + gid + 8 * up, c = nb * 8 + 2 * tig;
        uint32_t hi, lo;
        split2(S[nb][2 * up], S[nb][2 * up + 1], hi, lo);
        *reinterpret_cast<uint32_t*>(s_hi + row * kPitch + c) = hi;
        *reinterpret_cast<uint32_t*>(s_lo + row * kPitch + c) = lo;
      }
  };
  if (warp < SW) {
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
      for (int x = 0; x < 4; ++x)
        S[nb][x] = sp[(size_t)(col0 + nb * 8 + 2 * tig + (x & 1)) * DK + warp * 16 + gid + 8 * (x >> 1)];
    store_s();
  }
  const int arow = (lane & 7) + 8 * ((lane >> 3) & 1), achunk = lane >> 4;   // A operand, row-major
  const int trow = arow, tcol = 8 * (lane >> 4);                             // B operand whose k runs over rows

  const int chunks = (n + kChunk - 1) / kChunk;
  for (int ch = 0; ch < chunks; ++ch) {
    const int left = n - ch * kChunk;
    // this thread's places of u and o: rows wr * 16 + gid (+ 8), columns wc * 16 + 2 tig (+ 1, + 8, + 9)
    float u[2][4], o[2][4];
    const float* src = DELTA ? a.u : a.v;
#pragma unroll
    for (int up = 0; up < 2; ++up) {
      const int t = wr * 16 + gid + 8 * up;
      const float* row = src + ((size_t)(r0 + ch * kChunk + t) * a.H + h) * a.dv + col0 + wc * 16 + 2 * tig;
      const __nv_bfloat16* raw = a.raw.v + (size_t)(r0 + ch * kChunk + t) * a.raw.ld + h * a.dv + col0 + wc * 16 + 2 * tig;
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        const float2 x = t >= left ? make_float2(0.f, 0.f)
                         : RAW     ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(raw + nb * 8))
                                   : *reinterpret_cast<const float2*>(row + nb * 8);
        u[nb][2 * up] = x.x;
        u[nb][2 * up + 1] = x.y;
        o[nb][2 * up] = o[nb][2 * up + 1] = 0.f;
      }
    }
    float keep[2] = {0.f, 0.f};
    if (warp < SW) {
      const float* kp = a.keep + ((size_t)((r0 >> 6) + e + ch) * a.H + h) * DK + warp * 16 + gid;
      keep[0] = kp[0];
      keep[1] = kp[8];
    }
    cp_async_wait<0>();
    __syncthreads();   // q and w of this chunk and the memory before it are there; p and k of the last one are done with
    issue_write(ch);

    float d[2][4];   // W S0
#pragma unroll
    for (int nb = 0; nb < 2; ++nb) d[nb][0] = d[nb][1] = d[nb][2] = d[nb][3] = 0.f;
#pragma unroll(DELTA ? DK / 16 : 2)   // (delta rule, two at a time: 103.5 us, all eight 95.4; without: 43.0 / 43.5)
    for (int ks = 0; ks < DK / 16; ++ks) {
      uint32_t bh[4], bl[4], xh[4], xl[4];
      ldmatrix_x4_trans(bh[0], bh[1], bh[2], bh[3], smem_u32(s_hi + (ks * 16 + trow) * kPitch + wc * 16 + tcol));
      ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], smem_u32(s_lo + (ks * 16 + trow) * kPitch + wc * 16 + tcol));
      const int pos = swz<DK>(wr * 16 + arow, 2 * ks + achunk);
      if (DELTA) {
        ldmatrix_x4(xh[0], xh[1], xh[2], xh[3], smem_u32(w_s + pos));
        ldmatrix_x4(xl[0], xl[1], xl[2], xl[3], smem_u32(w_s + kChunk * DK + pos));
        mma3(d[0], xh, xl, bh[0], bh[1], bl[0], bl[1]);
        mma3(d[1], xh, xl, bh[2], bh[3], bl[2], bl[3]);
      }
      ldmatrix_x4(xh[0], xh[1], xh[2], xh[3], smem_u32(q_s + pos));
      ldmatrix_x4(xl[0], xl[1], xl[2], xl[3], smem_u32(q_s + kChunk * DK + pos));
      mma3(o[0], xh, xl, bh[0], bh[1], bl[0], bl[1]);
      mma3(o[1], xh, xl, bh[2], bh[3], bl[2], bl[3]);
    }
#pragma unroll
    for (int nb = 0; nb < 2; ++nb)
#pragma unroll
      for (int up = 0; up < 2; ++up) {
        uint32_t hi, lo;
        float x0 = u[nb][2 * up] - d[nb][2 * up], x1 = u[nb][2 * up + 1] - d[nb][2 * up + 1];
        if (!is_finite(largest(0.f, x0, x1))) {
          const int t = wr * 16 + gid + 8 * up, c = wc * 16 + nb * 8 + 2 * tig;
          bad_any = 1;
          if (!is_finite(x0)) atomicMin(&bad_col[c], t), x0 = 0.f;
          if (!is_finite(x1)) atomicMin(&bad_col[c + 1], t), x1 = 0.f;
        }
        split2(x0, x1, hi, lo);
        const int pos = (wr * 16 + gid + 8 * up) * kPitch + wc * 16 + nb * 8 + 2 * tig;
        *reinterpret_cast<uint32_t*>(u_hi + pos) = hi;
        *reinterpret_cast<uint32_t*>(u_lo + pos) = lo;
      }
    cp_async_wait<0>();
    __syncthreads();   // u, p and k are there; q, w and the memory's halves have been read
    const bool bad = bad_any != 0;
    if (ch + 1 < chunks) issue_read(ch + 1);

#pragma unroll
    for (int ks = 0; ks < kChunk / 16; ++ks) {   // o += P u: the keys of the runs up to the rows' own
      if (ks > wr) continue;
      uint32_t bh[4], bl[4], xh[4], xl[4];
      ldmatrix_x4_trans(bh[0], bh[1], bh[2], bh[3], smem_u32(u_hi + (ks * 16 + trow) * kPitch + wc * 16 + tcol));
      ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], smem_u32(u_lo + (ks * 16 + trow) * kPitch + wc * 16 + tcol));
      const int pos = swz<kChunk>(wr * 16 + arow, 2 * ks + achunk);
      ldmatrix_x4(xh[0], xh[1], xh[2], xh[3], smem_u32(p_s + pos));
      ldmatrix_x4(xl[0], xl[1], xl[2], xl[3], smem_u32(p_s + kChunk * kChunk + pos));
      mma3(o[0], xh, xl, bh[0], bh[1], bl[0], bl[1]);
      mma3(o[1], xh, xl, bh[2], bh[3], bl[2], bl[3]);
    }
    if (warp < SW) {   // S = e^{c_64} S + K^T u
#pragma unroll
      for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int x = 0; x < 4; ++x) S[nb][x] *= keep[x >> 1];
#pragma unroll
      for (int ks = 0; ks < kChunk / 16; ++ks) {
        uint32_t xh[4], xl[4];   // keys as the A operand, transposed: rows are key channels, k are tokens
        const int pos = swz<DK>(ks * 16 + (lane & 7) + 8 * (lane >> 4), warp * 2 + ((lane >> 3) & 1));
        ldmatrix_x4_trans(xh[0], xh[1], xh[2], xh[3], smem_u32(k_s + pos));
        ldmatrix_x4_trans(xl[0], xl[1], xl[2], xl[3], smem_u32(k_s + kChunk * DK + pos));
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          uint32_t bh[4], bl[4];
          ldmatrix_x4_trans(bh[0], bh[1], bh[2], bh[3], smem_u32(u_hi + (ks * 16 + trow) * kPitch + np * 16 + tcol));
          ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], smem_u32(u_lo + (ks * 16 + trow) * kPitch + np * 16 + tcol));
          mma3(S[2 * np], xh, xl, bh[0], bh[1], bl[0], bl[1]);
          mma3(S[2 * np + 1], xh, xl, bh[2], bh[3], bl[2], bl[3]);
        }
      }
      if (bad) {   // (for good: what the column's memory is multiplied by later stays NaN)
#pragma unroll
        for (int nb = 0; nb < 4; ++nb)
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (bad_col[nb * 8 + 2 * tig + (x & 1)] < kChunk) S[nb][x] = CUDART_NAN_F;
      }
      if (ch + 1 < chunks) store_s();
    }
    if (bad) {
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (bad_col[wc * 16 + nb * 8 + 2 * tig + (x & 1)] <= wr * 16 + gid + 8 * (x >> 1)) o[nb][x] = CUDART_NAN_F;
    }
#pragma unroll
    for (int up = 0; up < 2; ++up) {
      const int t = wr * 16 + gid + 8 * up;
      if (t >= left) continue;
      float* row = a.out + ((size_t)(r0 + ch * kChunk + t) * a.H + h) * a.dv + col0 + wc * 16 + 2 * tig;
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) *reinterpret_cast<float2*>(row + nb * 8) = make_float2(o[nb][2 * up], o[nb][2 * up + 1]);
    }
  }
  if (warp < SW) {
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
      for (int x = 0; x < 4; ++x)
        sp[(size_t)(col0 + nb * 8 + 2 * tig + (x & 1)) * DK + warp * 16 + gid + 8 * (x >> 1)] = S[nb][x];
  }
}

template <int DK, bool DELTA, bool HEAD, bool RAW = false>
int launch_chunked(const ChunkRows& a, int n_entries, int max_tokens, cudaStream_t stream) {
  auto prepare = chunk_prepare_kernel<DK, DELTA, HEAD, RAW>;
  auto walk = chunk_walk_kernel<DK, DELTA, RAW && !DELTA>;
  constexpr int prep_bytes = PrepShape<DK, DELTA, HEAD>::kBytes, walk_bytes = WalkShape<DK, DELTA>::kBytes;
  static_assert(walk_bytes <= 227 * 1024 && prep_bytes <= 227 * 1024, "shared memory of a block");
  static std::atomic<unsigned long long> prep_done{0}, walk_done{0};
  int rc = ccb_allow_smem(prepare, prep_bytes, prep_done);
  if (rc == 0) rc = ccb_allow_smem(walk, walk_bytes, walk_done);
  if (rc != 0) return rc;
  ccb_launch(prepare, dim3((max_tokens + kChunk - 1) / kChunk, a.H, n_entries), kThreads, prep_bytes, stream, a);
  rc = ccb_launch_status();
  if (rc != 0) return rc;
  ccb_launch(walk, dim3(a.dv / kCols, a.H, n_entries), kThreads, walk_bytes, stream, a);
  return ccb_launch_status();
}

}  // namespace

// Entries entry0 .. entry0 + n_entries - 1, the longest of max_tokens tokens.  Key sizes 64 and 128, value sizes that are
// multiples of 32 (others: CCB_REFUSE_SIZE).  q, k float [T, G, dk], v float [T, H, dv], g float [T, H, dk] (head_decay 0)
// or [T, H], beta float [T, H] (null: no delta rule).  Workspace: qs, ks and (delta rule) w [T, H, 2, dk] and p
// [T, H, 2, 64] bfloat16, u float [T, H, dv] (delta rule), keep float [T / 64 + entries, H, dk].  qs, ks, w and u may be
// the memory of q, k (where G = H), g (one decay per channel) and v: a block writes a row after it has read it, and
// nobody else reads it.  With the delta rule the decays per channel may come as the projection's bfloat16 rows a_rows, lda apart
// (see RawRows; g is not read then).
CCB_API int ccb_chunk_recurrence(const float* q, const float* k, const float* v, const float* g, const float* beta,
                                 const void* a_rows, int lda, const float* a_bias, const float* A_log, void* qs, void* ks, void* w, float* u, void* p, float* keep, float* state, float* out,
                                 const int* cu_q, const int* state_slot, int entry0, int n_entries, int max_tokens, int G, int H,
                                 int dk, int dv, int n_slots, int head_decay, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (G <= 0 || H <= 0 || H % G || (dk != 64 && dk != 128) || dv <= 0 || dv % kCols || entry0 < 0 || max_tokens <= 0 ||
      H > 65535 || n_entries > 65535)
    return CCB_REFUSE_SIZE;
  if (beta != nullptr && (w == nullptr || u == nullptr)) return CCB_REFUSE_ARG;
  if (a_rows != nullptr && (beta == nullptr || head_decay || a_bias == nullptr || A_log == nullptr)) return CCB_REFUSE_ARG;
  const auto bits = [](const void* x) { return reinterpret_cast<uintptr_t>(x); };
  if ((bits(q) | bits(k) | bits(v) | bits(g) | bits(qs) | bits(ks) | bits(w) | bits(u) | bits(p) | bits(out)) & 15)
    return CCB_REFUSE_ARG;
  if (G != H && (qs == (const void*)q || ks == (const void*)k)) return CCB_REFUSE_ARG;
  const ChunkRows a{q, k, v, g, beta, (__nv_bfloat16*)qs, (__nv_bfloat16*)ks, (__nv_bfloat16*)w, u, (__nv_bfloat16*)p, keep,
                    state, out, cu_q, state_slot, entry0, G, H, dv, n_slots,
                    RawRows{nullptr, nullptr, nullptr, (const __nv_bfloat16*)a_rows, 0, lda, a_bias, 0.f, 0.f, A_log}};
  if (a_rows != nullptr)
    return dk == 128 ? launch_chunked<128, true, false, true>(a, n_entries, max_tokens, stream)
                     : launch_chunked<64, true, false, true>(a, n_entries, max_tokens, stream);
#define CCB_CHUNK(DK, DELTA)                                                                \
  (head_decay ? launch_chunked<DK, DELTA, true>(a, n_entries, max_tokens, stream) \
              : launch_chunked<DK, DELTA, false>(a, n_entries, max_tokens, stream))
  if (dk == 128) return beta != nullptr ? CCB_CHUNK(128, true) : CCB_CHUNK(128, false);
  return beta != nullptr ? CCB_CHUNK(64, true) : CCB_CHUNK(64, false);
#undef CCB_CHUNK
}

// The form without the delta rule and with one decay per channel, from the projections' bfloat16 rows (see RawRows): q, k and v
// are the first columns of rows ld apart, on 8 bytes, a's rows lda apart.  Workspace as above.
CCB_API int ccb_chunk_recurrence_raw(const void* q, const void* k, const void* v, int ld, const void* a_rows, int lda,
                                     const float* bias, float q_mult, float tau, void* qs, void* ks, void* p, float* keep,
                                     float* state, float* out, const int* cu_q, const int* state_slot, int entry0, int n_entries,
                                     int max_tokens, int H, int dk, int dv, int n_slots, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (H <= 0 || (dk != 64 && dk != 128) || dv <= 0 || dv % kCols || entry0 < 0 || max_tokens <= 0 || H > 65535 ||
      n_entries > 65535 || ld % 4 || !(tau > 0.f))
    return CCB_REFUSE_SIZE;
  const auto bits = [](const void* x) { return reinterpret_cast<uintptr_t>(x); };
  if (((bits(qs) | bits(ks) | bits(p) | bits(out)) & 15) || ((bits(q) | bits(k) | bits(v)) & 7)) return CCB_REFUSE_ARG;
  const RawRows raw{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, (const __nv_bfloat16*)a_rows, ld, lda,
                    bias, q_mult, 1.0f / tau, nullptr};
  const ChunkRows a{nullptr, nullptr, nullptr, nullptr, nullptr, (__nv_bfloat16*)qs, (__nv_bfloat16*)ks, nullptr, nullptr,
                    (__nv_bfloat16*)p, keep, state, out, cu_q, state_slot, entry0, H, H, dv, n_slots, raw};
  return dk == 128 ? launch_chunked<128, false, false, true>(a, n_entries, max_tokens, stream)
                   : launch_chunked<64, false, false, true>(a, n_entries, max_tokens, stream);
}
