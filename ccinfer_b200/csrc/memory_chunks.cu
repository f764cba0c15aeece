// The recurrence of a matrix memory with one decay per head and token,
//
//   S <- a_t S + b_t k_t v_t^T;   o_t = S^T q_t * q_mult,
//
// over a request's portion of a prompt in chunks of 64 tokens on tensor cores (bfloat16 operands, float sums).  With
// c_t the sum of log a over the chunk up to t and S0 the memory before the chunk,
//
//   o_t = exp(c_t) S0^T q_t + sum_{s <= t} exp(c_t - c_s + log b_s) (q_t . k_s) v_s
//   S   = exp(c_64) S0 + sum_s exp(c_64 - c_s + log b_s) k_s v_s^T
//
// so a chunk is four small products, and only S is carried from chunk to chunk.  What the model computes in 32 bits
// stays so to about 2^-17: the logarithms and the exponentials are float, sums of logarithms are made in double and kept
// as two floats each (c_t - c_s of strong decays cancels: with 16 a token a single float left 1e-4 in the weight that a
// token gives itself, with 80 a token 9e-4); the memory lives in float registers for the whole portion; and every float
// that must become an operand (the memory, the weighted scores, the weighted values, queries and keys that were
// rotated) goes in as TWO bfloat16, its rounding and what the rounding left, each with a product of its own.  Queries,
// keys and values straight from a projection are bfloat16 already.
//
// A block: one request, one head, a slice of 8 NB value columns; four warps.  A warp takes 16 query rows of the chunk
// for the read-out and DK / 4 key channels of S for the update.  With a column of ones after the values (a running sum
// of the keys: n . q is one more column of o) the first slice takes it as one more block of eight columns.
// The next chunk's rows arrive through cp.async while this one is computed; two barriers a chunk.
//
// A state space layer's recurrence is the same with values that are floats (they enter as two bfloat16 as well) and with
// groups of heads that share queries and keys.  The two halves of queries and keys fill an SM's shared memory, so one block
// runs on it: of two teams of four warps, a slice of value columns each, that share the tiles of queries and keys and the
// weighted scores (a team makes those of every second block of 16 keys and leaves them for the other).  2,048 tokens of two
// requests, 128 heads of 64 x 128: 1,034 us token by token, 459 us in chunks by one team a block, 222 us by two.
// Outputs and memory are right to 5e-6 in the 2-norm, token by token to 2e-7; in a layer's results, whose rows are bfloat16
// (3.5e-3), neither shows.
// A value that is no finite number must not reach the tokens before it, whose weight of it is a zero that would still
// be multiplied by it: such a value enters the products as zero, and its column, from its token on, is made NaN
// afterwards.  (Values of 16 bits are multiplied where they lie: there it reaches up to 15 tokens before it.)
#include "common.cuh"
#include "mma_common.cuh"
#include <math_constants.h>

using namespace ccb;

namespace {

constexpr int kChunk = 64;
constexpr int kThreads = 128;   // of a team
constexpr int kGates = 5;       // numbers that a token's gates leave for a chunk
constexpr float kLeastLog = -200.f;   // a token's log decay at least: exp(-200) is zero in a float

struct ChunkArgs {
  const __nv_bfloat16 *q, *q_lo, *k, *k_lo, *v;
  const float* v32;           // float values in v's place
  int ldqk, ldv;              // row strides (q and k in one; q_lo, k_lo as q and k)
  int group;                  // neighbouring heads that share queries and keys
  const float* log_a;         // [tokens, H]
  const float* log_b;         // [tokens, H] or null: zero
  float* state;               // [slots, H, dvo, DK]
  float* out;                 // [tokens, H, dvo]
  const int *cu_q, *state_slot;
  int entry0, H, dv, dvo, max_slots;
  float q_mult;
};

// bfloat16 pair of (x, y) and of what their rounding left
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 f = __bfloat1622float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_bf16(x - f.x, y - f.y);
}

template <int DK, int NB, bool SPLIT, bool ONES, bool V32, int TEAMS>
__global__ void __launch_bounds__(kThreads * TEAMS)
memory_chunks_kernel(const ChunkArgs a) {
  static_assert(TEAMS == 1 || (V32 && TEAMS == 2), "two teams: with float values");
  ccb::pdl_begin();
  constexpr int BN = 8 * NB, VP = BN + 8;      // columns of the slice, pitch of its rows in shared memory (elements)
  constexpr int NT = NB + (ONES ? 1 : 0);      // blocks of eight columns
  constexpr int KS = DK / 16;
  constexpr int MT = DK / 64;                  // 16-row tiles of S a warp owns
  constexpr int TILE = kChunk * DK, VT = kChunk * VP;
  constexpr int QK = SPLIT ? 4 : 2;            // tiles of a stage: q, k (, their second halves)
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __nv_bfloat16* tiles = reinterpret_cast<__nv_bfloat16*>(smem_raw);   // [2][QK][64][DK], swizzled
  constexpr int TEAM = 4 * VT + 2 * DK * VP;                           // elements that a team has for itself
  const int team = threadIdx.x / kThreads;
  __nv_bfloat16* v_s = tiles + 2 * QK * TILE + team * TEAM;            // [2][64][VP] (V32: the values' two halves)
  __nv_bfloat16* s_hi = v_s + 2 * VT;                                  // [DK][VP]
  __nv_bfloat16* s_lo = s_hi + DK * VP;
  __nv_bfloat16* w_hi = s_lo + DK * VP;                                // [64][VP]
  __nv_bfloat16* w_lo = w_hi + VT;
  float* gates = reinterpret_cast<float*>(tiles + 2 * QK * TILE + TEAMS * TEAM);   // [2][kGates][64]: see write_gates
  uint4* p_s = reinterpret_cast<uint4*>(gates + 2 * kGates * kChunk);  // two teams: weighted scores, [10 tiles][2][32]
  // V32: by column of the slice, the first token of a chunk whose value is not finite (64: none); and whether there is one
  __shared__ int bad_col[V32 ? TEAMS * BN : 1], bad_any[TEAMS];

  const int e = a.entry0 + blockIdx.z, h = blockIdx.y, slice = blockIdx.x * TEAMS + team;
  const int slot = a.state_slot[e];
  const int r0 = a.cu_q[e], n = a.cu_q[e + 1] - r0;
  if (slot < 0 || slot >= a.max_slots || n <= 0) return;
  const int tid = threadIdx.x % kThreads, lane = tid & 31;   // in the team
  // Later rows of a chunk meet more keys: the second team's warps take theirs the other way round, so that each of an SM's four
  // schedulers has as much to do (the sizes above: 232 -> 222 us)
  const int warp = team == 0 ? tid >> 5 : 3 - (tid >> 5);
  const int gid = lane >> 2, tig = lane & 3;
  const int kvh = h / a.group;
  const int col0 = slice * BN;
  const bool ones = ONES && slice == 0;
  const int nt = NB + (ones ? 1 : 0);

  auto issue = [&](int chunk, int st) {
    const int t0 = chunk * kChunk;
    __nv_bfloat16* dst = tiles + st * QK * TILE;
    const __nv_bfloat16* src[4] = {a.q, a.k, a.q_lo, a.k_lo};
#pragma unroll
    for (int x = 0; x < QK; ++x)
#pragma unroll
      for (int i = 0; i < kChunk * (DK / 8) / (kThreads * TEAMS); ++i) {
        const int idx = threadIdx.x + kThreads * TEAMS * i;
        const int row = idx / (DK / 8), c = idx % (DK / 8);
        const bool ok = t0 + row < n;
        cp_async16(smem_u32(dst + x * TILE + swz<DK>(row, c)),
                   src[x] + (size_t)(r0 + t0 + (ok ? row : 0)) * a.ldqk + kvh * DK + c * 8, ok);
      }
    if constexpr (!V32) {
#pragma unroll
    for (int i = 0; i < (kChunk * NB + kThreads - 1) / kThreads; ++i) {
      const int idx = tid + kThreads * i;
      const int row = idx / NB, c = idx % NB;
      const bool ok = t0 + row < n;
      cp_async16(smem_u32(v_s + st * VT + row * VP + c * 8),
                 a.v + (size_t)(r0 + t0 + (ok ? row : 0)) * a.ldv + h * a.dv + col0 + c * 8, ok);
    }
    }
    cp_async_commit();
  };

  // V32: half a row of the slice a thread, loaded one chunk ahead
  float4 vv[V32 ? NB : 1];
  auto load_values = [&](int chunk) {
    const int t = chunk * kChunk + (tid >> 1);
    const float4* src = reinterpret_cast<const float4*>(a.v32 + (size_t)(r0 + t) * a.ldv + h * a.dv + col0 + (tid & 1) * (BN / 2));
#pragma unroll
    for (int c = 0; c < NB; ++c) vv[c] = t < n ? src[c] : make_float4(0.f, 0.f, 0.f, 0.f);
  };

  // The gates of a chunk, two tokens a lane of warp 0: loaded one chunk ahead, summed and left in shared memory.
  float la[2], lb[2];
  auto load_gates = [&](int chunk) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = chunk * kChunk + 2 * lane + i;
      const bool ok = t < n;
      const float x = ok ? a.log_a[(size_t)(r0 + t) * a.H + h] : 0.f;
      la[i] = x < kLeastLog ? kLeastLog : x;
      lb[i] = ok ? (a.log_b ? a.log_b[(size_t)(r0 + t) * a.H + h] : 0.f) : -CUDART_INF_F;
    }
  };
  // c_t (its float and what that left), exp(c_t), log b_t, exp(c_64 - c_t) b_t
  auto write_gates = [&](int st) {
    float* g = gates + st * kGates * kChunk + 2 * lane;
    double sum = (double)la[0] + (double)la[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double p = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += p;
    }
    const double total = __shfl_sync(0xffffffffu, sum, 31);
    double before = __shfl_up_sync(0xffffffffu, sum, 1);
    if (lane == 0) before = 0.;
    const double c[2] = {before + (double)la[0], sum};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float hi = (float)c[i];
      g[i] = hi;
      g[kChunk + i] = (float)(c[i] - (double)hi);
      g[2 * kChunk + i] = expf(hi);
      g[3 * kChunk + i] = lb[i];
      g[4 * kChunk + i] = expf((float)(total - c[i]) + lb[i]);
    }
  };

  issue(0, 0);
  if constexpr (V32) {
    load_values(0);
    if (tid < BN) bad_col[team * BN + tid] = kChunk;
    if (tid == 0) bad_any[team] = 0;
  }
  const bool gating = warp == 0 && team == 0;
  if (gating) {
    load_gates(0);
    write_gates(0);
    load_gates(1);
  }
  // the column of ones beside the values (and zeros after it): the same in both stages, for good
  if constexpr (!V32)   // (V32 has no such column)
    for (int i = tid; i < 2 * kChunk * 8; i += kThreads)
      v_s[(i >> 3) * VP + BN + (i & 7)] = __float2bfloat16_rn((i & 7) == 0 && ones ? 1.f : 0.f);
  for (int i = tid; i < kChunk * 8; i += kThreads) {
    w_hi[(i >> 3) * VP + BN + (i & 7)] = __float2bfloat16_rn(0.f);
    w_lo[(i >> 3) * VP + BN + (i & 7)] = __float2bfloat16_rn(0.f);
  }

  // S: rows (key channels) m0 .. of the warp, columns of the slice; the accumulator layout of the update's product
  float S[MT][NT][4];
  float* sp = a.state + ((size_t)slot * a.H + h) * a.dvo * DK;
  auto column = [&](int nb, int c) { return nb < NB ? col0 + nb * 8 + c : (c == 0 ? a.dv : -1); };
  auto store_s = [&]() {   // the memory as two bfloat16, rows of key channels
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nb = 0; nb < NT; ++nb) {
        if (nb >= nt) continue;
        const int row = (warp * MT + mt) * 16 + gid, c = nb * 8 + 2 * tig;
        uint32_t hi, lo;
        split2(S[mt][nb][0], S[mt][nb][1], hi, lo);
        *reinterpret_cast<uint32_t*>(s_hi + row * VP + c) = hi;
        *reinterpret_cast<uint32_t*>(s_lo + row * VP + c) = lo;
        split2(S[mt][nb][2], S[mt][nb][3], hi, lo);
        *reinterpret_cast<uint32_t*>(s_hi + (row + 8) * VP + c) = hi;
        *reinterpret_cast<uint32_t*>(s_lo + (row + 8) * VP + c) = lo;
      }
  };
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nb = 0; nb < NT; ++nb)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int row = (warp * MT + mt) * 16 + gid + 8 * (x >> 1);
        const int c = nb < nt ? column(nb, 2 * tig + (x & 1)) : -1;
        S[mt][nb][x] = c >= 0 ? sp[(size_t)c * DK + row] : 0.f;
      }
  store_s();

  // rows of an operand whose k runs over rows of shared memory with pitch VP: block pair p (16 columns), 16 k from k0;
  // the last single block reads its own columns twice
  const int trow = (lane & 7) + 8 * ((lane >> 3) & 1);
  auto load_b = [&](const __nv_bfloat16* base, int k0, int nb, bool single, uint32_t* b) {
    const int c = nb * 8 + (single ? 0 : 8 * (lane >> 4));
    ldmatrix_x4_trans(b[0], b[1], b[2], b[3], smem_u32(base + (k0 + trow) * VP + c));
  };

  const int chunks = (n + kChunk - 1) / kChunk;
  for (int ch = 0; ch < chunks; ++ch) {
    const int st = ch & 1;
    cp_async_wait<0>();
    __syncthreads();   // the chunk's rows and gates are there; everybody is done with the chunk before
    if (ch + 1 < chunks) issue(ch + 1, st ^ 1);
    if (gating && ch + 1 < chunks) {
      write_gates(st ^ 1);
      load_gates(ch + 2);
    }
    const __nv_bfloat16 *qt = tiles + st * QK * TILE, *kt = qt + TILE, *ql = qt + 2 * TILE, *kl = qt + 3 * TILE;
    const __nv_bfloat16* vt = v_s + (V32 ? 0 : st * VT);
    const float *gc = gates + st * kGates * kChunk, *gl = gc + kChunk, *ga = gl + kChunk, *gb = ga + kChunk, *gw = gb + kChunk;

    {   // the values times their weights in the chunk's contribution to S
      const int row = tid >> 1, part = (tid & 1) * (BN / 2);
      const float w = gw[row];
      if constexpr (V32) {
        float most = 0.f;
#pragma unroll
        for (int c = 0; c < NB; ++c) most = largest(largest(most, vv[c].x, vv[c].y), vv[c].z, vv[c].w);
        if (!is_finite(most)) {
          bad_any[team] = 1;
#pragma unroll
          for (int c = 0; c < BN / 2; ++c) {
            float& x = c % 4 == 0 ? vv[c / 4].x : c % 4 == 1 ? vv[c / 4].y : c % 4 == 2 ? vv[c / 4].z : vv[c / 4].w;
            if (!is_finite(x)) {
              atomicMin(&bad_col[team * BN + part + c], row);
              x = 0.f;
            }
          }
        }
#pragma unroll
        for (int c = 0; c < BN / 2; c += 2) {
          const float2 f = c & 2 ? make_float2(vv[c / 4].z, vv[c / 4].w) : make_float2(vv[c / 4].x, vv[c / 4].y);
          uint32_t hi, lo;
          split2(f.x, f.y, hi, lo);
          *reinterpret_cast<uint32_t*>(v_s + row * VP + part + c) = hi;
          *reinterpret_cast<uint32_t*>(v_s + VT + row * VP + part + c) = lo;
          split2(f.x * w, f.y * w, hi, lo);
          *reinterpret_cast<uint32_t*>(w_hi + row * VP + part + c) = hi;
          *reinterpret_cast<uint32_t*>(w_lo + row * VP + part + c) = lo;
        }
        if (ch + 1 < chunks) load_values(ch + 1);
      } else {
#pragma unroll
      for (int c = 0; c < BN / 2; c += 2) {
        const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(vt + row * VP + part + c);
        const float2 f = __bfloat1622float2(x);
        uint32_t hi, lo;
        split2(f.x * w, f.y * w, hi, lo);
        *reinterpret_cast<uint32_t*>(w_hi + row * VP + part + c) = hi;
        *reinterpret_cast<uint32_t*>(w_lo + row * VP + part + c) = lo;
      }
      }
      if (ones && (tid & 1) == 0) {
        const __nv_bfloat16 hi = __float2bfloat16_rn(w);
        w_hi[row * VP + BN] = hi;
        w_lo[row * VP + BN] = __float2bfloat16_rn(w - __bfloat162float(hi));
      }
    }

    // read-out of rows warp * 16 ..: first S0^T q and the raw scores q . k of the keys up to the rows' own block
    // (two teams: of every second block of keys each)
    constexpr int NP = 4 / TEAMS;
    float acc[NT][4], s[2 * NP][4];
#pragma unroll
    for (int nb = 0; nb < NT; ++nb) acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.f;
#pragma unroll
    for (int i = 0; i < 2 * NP; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
    const int arow = warp * 16 + (lane & 7) + 8 * ((lane >> 3) & 1), achunk = lane >> 4;
    const int krow = (lane & 7) + 8 * (lane >> 4), kchunk = (lane >> 3) & 1;
#pragma unroll 2
    for (int ks = 0; ks < KS; ++ks) {
      uint32_t qa[4], qb[4];
      ldmatrix_x4(qa[0], qa[1], qa[2], qa[3], smem_u32(qt + swz<DK>(arow, 2 * ks + achunk)));
      if (SPLIT) ldmatrix_x4(qb[0], qb[1], qb[2], qb[3], smem_u32(ql + swz<DK>(arow, 2 * ks + achunk)));
#pragma unroll
      for (int nb = 0; nb < NT; nb += 2) {
        if (nb >= nt) continue;
        const bool single = nb + 1 >= NT;
        uint32_t bh[4], bl[4];
        load_b(s_hi, ks * 16, nb, single, bh);
        load_b(s_lo, ks * 16, nb, single, bl);
        mma_bf16_16816(acc[nb], qa, bh[0], bh[1]);
        mma_bf16_16816(acc[nb], qa, bl[0], bl[1]);
        if (SPLIT) mma_bf16_16816(acc[nb], qb, bh[0], bh[1]);
        if (!single) {
          mma_bf16_16816(acc[nb + 1 < NT ? nb + 1 : nb], qa, bh[2], bh[3]);
          mma_bf16_16816(acc[nb + 1 < NT ? nb + 1 : nb], qa, bl[2], bl[3]);
          if (SPLIT) mma_bf16_16816(acc[nb + 1 < NT ? nb + 1 : nb], qb, bh[2], bh[3]);
        }
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int np = TEAMS * p + (TEAMS > 1 ? team : 0);
        if (np > warp) continue;
        uint32_t b[4];
        ldmatrix_x4(b[0], b[1], b[2], b[3], smem_u32(kt + swz<DK>(np * 16 + krow, 2 * ks + kchunk)));
        mma_bf16_16816(s[2 * p], qa, b[0], b[1]);
        mma_bf16_16816(s[2 * p + 1], qa, b[2], b[3]);
        if (SPLIT) {
          mma_bf16_16816(s[2 * p], qb, b[0], b[1]);
          mma_bf16_16816(s[2 * p + 1], qb, b[2], b[3]);
          ldmatrix_x4(b[0], b[1], b[2], b[3], smem_u32(kl + swz<DK>(np * 16 + krow, 2 * ks + kchunk)));
          mma_bf16_16816(s[2 * p], qa, b[0], b[1]);
          mma_bf16_16816(s[2 * p + 1], qa, b[2], b[3]);
        }
      }
    }
    if (V32 && TEAMS == 1) __syncthreads();   // the values' halves are complete
    const int t_lo = warp * 16 + gid, t_hi = t_lo + 8;
    const float a_lo = ga[t_lo] * a.q_mult, a_hi = ga[t_hi] * a.q_mult;
    const float c_lo = gc[t_lo], c_hi = gc[t_hi], cl_lo = gl[t_lo], cl_hi = gl[t_hi];
#pragma unroll
    for (int nb = 0; nb < NT; ++nb) {
      acc[nb][0] *= a_lo; acc[nb][1] *= a_lo;
      acc[nb][2] *= a_hi; acc[nb][3] *= a_hi;
    }
    // weights of a block of 16 keys, times its scores, as two bfloat16
    auto weigh = [&](int np, float (*sc)[4], uint32_t* ph, uint32_t* pl) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float* x = sc[half];
        const int j = np * 16 + half * 8 + 2 * tig;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const float c = gc[j + y], l = gl[j + y], b = gb[j + y];
          x[y] = j + y <= t_lo ? x[y] * (expf(((c_lo - c) + (cl_lo - l)) + b) * a.q_mult) : 0.f;
          x[2 + y] = j + y <= t_hi ? x[2 + y] * (expf(((c_hi - c) + (cl_hi - l)) + b) * a.q_mult) : 0.f;
        }
        split2(x[0], x[1], ph[2 * half], pl[2 * half]);
        split2(x[2], x[3], ph[2 * half + 1], pl[2 * half + 1]);
      }
    };
    auto weighted_values = [&](int np, const uint32_t* ph, const uint32_t* pl) {
#pragma unroll
      for (int nb = 0; nb < NT; nb += 2) {
        if (nb >= nt) continue;
        const bool single = nb + 1 >= NT;
        uint32_t b[4];
        load_b(vt, np * 16, nb, single, b);
        mma_bf16_16816(acc[nb], ph, b[0], b[1]);
        mma_bf16_16816(acc[nb], pl, b[0], b[1]);
        if (!single) {
          mma_bf16_16816(acc[nb + 1 < NT ? nb + 1 : nb], ph, b[2], b[3]);
          mma_bf16_16816(acc[nb + 1 < NT ? nb + 1 : nb], pl, b[2], b[3]);
        }
        if constexpr (V32) {
          load_b(vt + VT, np * 16, nb, single, b);
          mma_bf16_16816(acc[nb], ph, b[0], b[1]);
          if (!single) mma_bf16_16816(acc[nb + 1 < NT ? nb + 1 : nb], ph, b[2], b[3]);
        }
      }
    };
    if constexpr (TEAMS == 1) {
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        if (np > warp) continue;
        uint32_t ph[4], pl[4];
        weigh(np, s + 2 * np, ph, pl);
        weighted_values(np, ph, pl);
      }
    } else {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int np = 2 * p + team;
        if (np > warp) continue;
        uint32_t ph[4], pl[4];
        weigh(np, s + 2 * p, ph, pl);
        uint4* to = p_s + (warp * (warp + 1) / 2 + np) * 64 + lane;
        to[0] = make_uint4(ph[0], ph[1], ph[2], ph[3]);
        to[32] = make_uint4(pl[0], pl[1], pl[2], pl[3]);
      }
      __syncthreads();   // the weighted scores and both forms of the values are complete, and everybody has read S0
      for (int np = 0; np <= warp; ++np) {
        const uint4* from = p_s + (warp * (warp + 1) / 2 + np) * 64 + lane;
        const uint4 x = from[0], y = from[32];
        const uint32_t ph[4] = {x.x, x.y, x.z, x.w}, pl[4] = {y.x, y.y, y.z, y.w};
        weighted_values(np, ph, pl);
      }
    }
    // (the barrier before the weighted values has passed)
    const bool bad = V32 && bad_any[team] != 0;
    if (V32 && bad) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (bad_col[team * BN + nb * 8 + 2 * tig + (x & 1)] <= (x < 2 ? t_lo : t_hi)) acc[nb][x] = CUDART_NAN_F;
    }
    const int left = n - ch * kChunk;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int t = x == 0 ? t_lo : t_hi;
      if (t < left) {
        float* o = a.out + ((size_t)(r0 + ch * kChunk + t) * a.H + h) * a.dvo;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          o[col0 + nb * 8 + 2 * tig] = acc[nb][2 * x];
          o[col0 + nb * 8 + 2 * tig + 1] = acc[nb][2 * x + 1];
        }
        if (ones && tig == 0) o[a.dv] = acc[NT - 1][2 * x];
      }
    }
    if constexpr (TEAMS == 1) __syncthreads();   // everybody has read S0, and the weighted values are complete

    const float keep = ga[kChunk - 1];   // exp(c_64)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nb = 0; nb < NT; ++nb)
#pragma unroll
        for (int x = 0; x < 4; ++x) S[mt][nb][x] *= keep;
#pragma unroll
    for (int ks = 0; ks < kChunk / 16; ++ks) {
      // keys as the A operand, transposed: rows are key channels, k are tokens
      uint32_t ka[MT][4], kb[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int token = ks * 16 + (lane & 7) + 8 * (lane >> 4);
        const int c8 = (warp * MT + mt) * 2 + ((lane >> 3) & 1);
        ldmatrix_x4_trans(ka[mt][0], ka[mt][1], ka[mt][2], ka[mt][3], smem_u32(kt + swz<DK>(token, c8)));
        if (SPLIT) ldmatrix_x4_trans(kb[mt][0], kb[mt][1], kb[mt][2], kb[mt][3], smem_u32(kl + swz<DK>(token, c8)));
      }
#pragma unroll
      for (int nb = 0; nb < NT; nb += 2) {
        if (nb >= nt) continue;
        const bool single = nb + 1 >= NT;
        uint32_t bh[4], bl[4];
        load_b(w_hi, ks * 16, nb, single, bh);
        load_b(w_lo, ks * 16, nb, single, bl);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          mma_bf16_16816(S[mt][nb], ka[mt], bh[0], bh[1]);
          mma_bf16_16816(S[mt][nb], ka[mt], bl[0], bl[1]);
          if (SPLIT) mma_bf16_16816(S[mt][nb], kb[mt], bh[0], bh[1]);
          if (!single) {
            mma_bf16_16816(S[mt][nb + 1 < NT ? nb + 1 : nb], ka[mt], bh[2], bh[3]);
            mma_bf16_16816(S[mt][nb + 1 < NT ? nb + 1 : nb], ka[mt], bl[2], bl[3]);
            if (SPLIT) mma_bf16_16816(S[mt][nb + 1 < NT ? nb + 1 : nb], kb[mt], bh[2], bh[3]);
          }
        }
      }
    }
    if (V32 && bad) {   // (for good: what the column's memory is multiplied by later stays NaN)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (bad_col[team * BN + nb * 8 + 2 * tig + (x & 1)] < kChunk) S[mt][nb][x] = CUDART_NAN_F;
    }
    if (ch + 1 < chunks) store_s();
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nb = 0; nb < NT; ++nb)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int row = (warp * MT + mt) * 16 + gid + 8 * (x >> 1);
        const int c = nb < nt ? column(nb, 2 * tig + (x & 1)) : -1;
        if (c >= 0) sp[(size_t)c * DK + row] = S[mt][nb][x];
      }
}

template <int DK, int NB, bool SPLIT, bool ONES, bool V32 = false, int TEAMS = 1>
int launch_chunks(const ChunkArgs& a, int n_entries, cudaStream_t stream) {
  constexpr int VP = 8 * NB + 8;
  constexpr size_t smem = (size_t)(2 * (SPLIT ? 4 : 2) * kChunk * DK + TEAMS * (4 * kChunk * VP + 2 * DK * VP)) * 2 +
                          2 * kGates * kChunk * sizeof(float) + (TEAMS > 1 ? 10 * 2 * 32 * sizeof(uint4) : 0);
  static_assert(smem <= 227 * 1024, "shared memory of a block");
  const auto kernel = memory_chunks_kernel<DK, NB, SPLIT, ONES, V32, TEAMS>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  ccb_launch(kernel, dim3(a.dv / (8 * NB * TEAMS), a.H, n_entries), dim3(kThreads * TEAMS), smem, stream, a);
  return ccb_launch_status();
}

template <int DK, int NB>
int pick_chunks(const ChunkArgs& a, int n_entries, cudaStream_t stream) {
  const bool split = a.q_lo != nullptr, ones = a.dvo > a.dv;
  if (split) return ones ? launch_chunks<DK, NB, true, true>(a, n_entries, stream) : launch_chunks<DK, NB, true, false>(a, n_entries, stream);
  return ones ? launch_chunks<DK, NB, false, true>(a, n_entries, stream) : launch_chunks<DK, NB, false, false>(a, n_entries, stream);
}

}  // namespace

// Key sizes 64 and 128, value sizes that are multiples of 16 (others: CCB_REFUSE_SIZE).  q, k (and q_lo, k_lo: what the
// rounding of q and k to bfloat16 left, or null) [tokens, ldqk] with head h at column h * dk; v [tokens, ldv] with head
// h at column h * dv; log_a, log_b (null: zero) float [tokens, H]; state float [slots, H, dvo, dk] and out float
// [tokens, H, dvo] with dvo = dv, or dv + 1 for a last value column of ones.  Entries entry0 .. entry0 + n_entries - 1.
CCB_API int ccb_memory_chunks(const void* q, const void* q_lo, const void* k, const void* k_lo, int ldqk, const void* v,
                              int ldv, const float* log_a, const float* log_b, float* state, float* out, const int* cu_q,
                              const int* state_slot, int entry0, int n_entries, int H, int dk, int dv, int dvo,
                              int max_slots, float q_mult, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (H <= 0 || (dk != 64 && dk != 128) || dv <= 0 || dv % 16 || (dvo != dv && dvo != dv + 1) || ldqk % 8 || ldv % 8)
    return CCB_REFUSE_SIZE;
  if ((q_lo == nullptr) != (k_lo == nullptr) || log_a == nullptr) return CCB_REFUSE_ARG;
  const auto bits = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  if ((bits(q) | bits(q_lo) | bits(k) | bits(k_lo) | bits(v)) & 15) return CCB_REFUSE_ARG;
  const __nv_bfloat16 *qp = (const __nv_bfloat16*)q, *qlp = (const __nv_bfloat16*)q_lo, *kp = (const __nv_bfloat16*)k,
                      *klp = (const __nv_bfloat16*)k_lo, *vp = (const __nv_bfloat16*)v;
  const ChunkArgs a{qp, qlp, kp, klp, vp, nullptr, ldqk, ldv, 1, log_a, log_b, state, out, cu_q, state_slot, entry0, H, dv, dvo,
                    max_slots, q_mult};
  // slices of 32 columns where they give enough blocks, else of 16
  const bool wide = dv % 32 == 0 && (long long)(dv / 32) * H * n_entries >= 96;
  if (dk == 128) return wide ? pick_chunks<128, 4>(a, n_entries, stream) : pick_chunks<128, 2>(a, n_entries, stream);
  return wide ? pick_chunks<64, 4>(a, n_entries, stream) : pick_chunks<64, 2>(a, n_entries, stream);
}

// The same for a state space layer: values float [tokens, H, P] (their rows ldv apart), queries and keys of G groups of N
// coordinates [tokens, ldqk] as two bfloat16 each; N 64 or 128, P a multiple of 16.
CCB_API int ccb_ssm_chunks(const void* q, const void* q_lo, const void* k, const void* k_lo, int ldqk, const float* v, int ldv,
                           const float* log_a, const float* log_b, float* state, float* out, const int* cu_q,
                           const int* state_slot, int entry0, int n_entries, int G, int H, int N, int P, int max_slots,
                           cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  if (G <= 0 || H <= 0 || H % G || (N != 64 && N != 128) || P <= 0 || P % 16 || ldqk % 8 || ldv % 4) return CCB_REFUSE_SIZE;
  if (q_lo == nullptr || k_lo == nullptr || log_a == nullptr) return CCB_REFUSE_ARG;
  const auto bits = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  if ((bits(q) | bits(q_lo) | bits(k) | bits(k_lo) | bits(v)) & 15) return CCB_REFUSE_ARG;
  const ChunkArgs a{(const __nv_bfloat16*)q, (const __nv_bfloat16*)q_lo, (const __nv_bfloat16*)k, (const __nv_bfloat16*)k_lo,
                    nullptr, v, ldqk, ldv, H / G, log_a, log_b, state, out, cu_q, state_slot, entry0, H, P, P, max_slots, 1.f};
  // Two teams where P is a multiple of 32, of 32 columns each where that gives half the SMs a block, else (the walk of a request
  // is a serial chain, and narrower slices have more SMs at it) of 16; one team of 16 for other P.
  const bool wide = P % 64 == 0 && (long long)(P / 64) * H * n_entries >= 74;
#define CCB_SSM_CHUNKS(DK)                                                               \
  return wide          ? launch_chunks<DK, 4, true, false, true, 2>(a, n_entries, stream) \
         : P % 32 == 0 ? launch_chunks<DK, 2, true, false, true, 2>(a, n_entries, stream) \
                       : launch_chunks<DK, 2, true, false, true, 1>(a, n_entries, stream)
  if (N == 128) CCB_SSM_CHUNKS(128);
  CCB_SSM_CHUNKS(64);
#undef CCB_SSM_CHUNKS
}
