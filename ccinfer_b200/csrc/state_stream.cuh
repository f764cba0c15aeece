// One token each of many requests through a recurrence with a matrix per (request, head):
//
//   S <- g S;  u = beta (v - S^T k) (the delta rule) or beta v;  S <- S + k u^T;  o = S^T q
//
// which is a stream of the states, read and written once.  A block an SM walks over (request, head); a head's whole state
// (dv x dk floats, at most 64 KB) is one bulk copy into a ring of shared memory and one back out of it, so that the memory
// always has one state on its way in and one on its way out while a third is worked on:
//
//   warp 0       the copies: a state in as soon as a place is free; one out, from where it lay, when it has been computed
//   warps 1 - 6  two teams of three that make q, k, v and the gates of a state in turn (`Job::prepare`), up to four ahead
//   warps 7 - 14 the recurrence: a warp eight or sixteen neighbouring value channels, four key channels a lane
//
// Bound by memory (48 requests of 32 heads of 128 x 128, 201 MB: 40 us, 5.0 TB/s).  A block that loads its state into
// registers, computes and stores it, two to an SM, waits for one thing after the other: 67 us so.  A layer, before / with the
// stream, us, 48, 16 and 8 requests: one decay a head (32 heads of 128 x 128) 112 / 86, 76 / 72, 61 / 53; one a channel
// 145 / 100, 89 / 76, 72 / 66; gated linear attention 130 / 85, 86 / 72, 62 / 55; state space (128 heads of 64 x 128) 185 /
// 133, 115 / 96, 87 / 78.
#pragma once

#include "common.cuh"
#include "tc_common.cuh"

namespace ccb {

constexpr int kStreamTeams = 2, kStreamTeamWarps = 3, kStreamWarps = 8;
constexpr int kStreamThreads = 32 * (1 + kStreamTeams * kStreamTeamWarps + kStreamWarps);
constexpr int kStreamAhead = 4;      // states whose rows are ready or being made
constexpr int kStreamDim = 128;      // key and value channels at most
constexpr int kStreamBytes = 192 * 1024;   // of states
constexpr int kStreamStages = 12;    // at most

// What a team leaves for the warps of the recurrence.  Beyond dk and dv: zeros.
struct StreamRows {
  float q[kStreamDim], k[kStreamDim], g[kStreamDim], v[kStreamDim], w[kStreamDim];   // g: with a decay per channel; w: of the output
  float decay, beta, pad[2];
};

struct StateStream {
  float* state;              // [slots, H, dv, dk]
  const int *state_slot, *cu_q;
  int n_slots, n_entries, H, dk, dv, stages;
  int* status;
};

// bytes (a multiple of 16) side by side, both ends on 16 bytes
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ float stream_dot4(const float4 a, const float4 b) { return (a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w); }

// Job: prepare(part, lane, t, e, h, slot, rows, wait): part 0, 1, 2 of a team's work for token row t (a warp each), which
//      loads, calls wait() and, if that is true, writes to rows;
//      DELTA, CHANNEL (a decay per key channel), NORM (o / rms(o) * w is what is stored);  store(t, h, c, value), eps;
//      AHEAD: the copies may begin while the kernel ahead in the stream still runs, which then must not write the states or
//      the step's tables (that kernel is the projection of this one's rows; a second call on the same states would have to wait).
// U: value channels of a warp, 8 or 16.
template <class Job, int U>
__global__ void __launch_bounds__(kStreamThreads, 1)
state_stream_kernel(const StateStream a, const Job job) {
  extern __shared__ __align__(128) uint8_t stream_smem[];
  __shared__ __align__(16) StreamRows rows_s[kStreamAhead];
  __shared__ __align__(8) uint64_t bars[2 * kStreamStages + 2 * kStreamAhead];
  __shared__ float* home[kStreamStages];   // where a stage's state lies
  __shared__ float red[2][kStreamWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = s32(bars), done0 = full0 + 8 * kStreamStages, ready0 = done0 + 8 * kStreamStages,
                 taken0 = ready0 + 8 * kStreamAhead;
  const int size = a.dv * a.dk, items = a.n_entries * a.H;
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(done0 + 8 * s, kStreamWarps);
    }
    for (int s = 0; s < kStreamAhead; ++s) {
      mbar_init(ready0 + 8 * s, kStreamTeamWarps);
      mbar_init(taken0 + 8 * s, kStreamWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto slot_of = [&](int e) {
    const int slot = a.state_slot[e];
    return slot < a.n_slots ? slot : -1;
  };
  auto give_up = [&]() { set_status(a.status, CCB_ST_WAIT_TIMEOUT); };

  if (warp == 0) {
    if (lane == 0) {
      if (!Job::AHEAD) pdl_wait();
      auto out = [&](int n) {   // the state of item n, once it has been computed
        const int s = n % a.stages;
        if (!mbar_wait(done0 + 8 * s, (n / a.stages) & 1)) {
          give_up();
          return false;
        }
        bulk_store(home[s], s32(stream_smem) + s * size * 4, size * 4);
        return true;
      };
      int n = 0;
      bool alive = true;
      for (int item = blockIdx.x; item < items && alive; item += gridDim.x) {
        const int e = item / a.H, h = item - e * a.H, slot = slot_of(e), s = n % a.stages;
        if (slot < 0) continue;
        if (n >= a.stages) {
          alive = out(n - a.stages);
          if (!alive) break;
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        home[s] = a.state + ((size_t)slot * a.H + h) * size;
        mbar_expect_tx(full0 + 8 * s, size * 4);
        bulk_load(s32(stream_smem) + s * size * 4, home[s], size * 4, full0 + 8 * s);
        ++n;
      }
      for (int m = n > a.stages ? n - a.stages : 0; m < n && alive; ++m) alive = out(m);
      if (!alive)   // no copy may land after the block has gone
        for (int m = n > a.stages ? n - a.stages : 0; m < n; ++m) mbar_wait(full0 + 8 * (m % a.stages), (m / a.stages) & 1);
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    return;
  }
  pdl_wait();
  if (threadIdx.x == 32) pdl_trigger();
  if (warp <= kStreamTeams * kStreamTeamWarps) {
    const int team = (warp - 1) / kStreamTeamWarps, part = (warp - 1) % kStreamTeamWarps;
    int n = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int e = item / a.H, h = item - e * a.H, slot = slot_of(e);
      if (slot < 0) continue;
      const int place = n % kStreamAhead, turn = n / kStreamAhead;
      const bool mine = n++ % kStreamTeams == team;
      if (!mine) continue;
      const bool ok = job.prepare(part, lane, a.cu_q[e], e, h, slot, rows_s[place],
                                  [&]() { return __all_sync(0xffffffffu, mbar_wait(taken0 + 8 * place, (turn & 1) ^ 1)) != 0; });
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(ready0 + 8 * place);
    }
    return;
  }
  // ---- the recurrence: value channels c0 .. c0 + U - 1 of the warp, key channels 4 lane ..
  const int w = warp - 1 - kStreamTeams * kStreamTeamWarps, c0 = w * U;
  const bool on = 4 * lane < a.dk;
  // after the sums a lane has one channel's: with sixteen k's product in the lower half, q's in the upper one, with eight
  // every channel twice
  constexpr int kHold = 16 / U;
  const int mine = c0 + (lane & 15) / kHold;
  const bool has = mine < a.dv && lane < 16 && lane % kHold == 0;
  int n = 0;
  bool alive = true;   // (a warp that gave up still meets the others at the barrier below)
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int e = item / a.H, h = item - e * a.H;
    if (slot_of(e) < 0) continue;
    const int s = n % a.stages, place = n % kStreamAhead, t = a.cu_q[e];
    if (alive) {
      alive = __all_sync(0xffffffffu, mbar_wait(ready0 + 8 * place, (n / kStreamAhead) & 1) && mbar_wait(full0 + 8 * s, (n / a.stages) & 1));
      if (!alive && lane == 0) give_up();
    }
    float o = 0.f, ww = 0.f;
    if (alive) {
      const StreamRows& rows = rows_s[place];
      const float4 kk = *reinterpret_cast<const float4*>(rows.k + 4 * lane), qq = *reinterpret_cast<const float4*>(rows.q + 4 * lane);
      float4 g;
      if (Job::CHANNEL) g = *reinterpret_cast<const float4*>(rows.g + 4 * lane);
      else g.x = g.y = g.z = g.w = rows.decay;
      const float beta = rows.beta, v = mine < a.dv ? rows.v[mine] : 0.f;
      if (Job::NORM && mine < a.dv) ww = rows.w[mine];
      float* S = reinterpret_cast<float*>(stream_smem) + (size_t)s * size + c0 * a.dk + 4 * lane;
      float4 z[U];
      float m[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        z[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (on && c0 + u < a.dv) z[u] = *reinterpret_cast<const float4*>(S + u * a.dk);
      }
      const float kq = warp_sum(stream_dot4(kk, qq));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        z[u].x *= g.x; z[u].y *= g.y; z[u].z *= g.z; z[u].w *= g.w;
        const float dotk = Job::DELTA ? stream_dot4(z[u], kk) : 0.f, dotq = stream_dot4(z[u], qq);
        m[u] = (lane & 16 ? dotq : dotk) + __shfl_xor_sync(0xffffffffu, lane & 16 ? dotk : dotq, 16);
      }
#pragma unroll
      for (int x = U / 2; x > 0; x >>= 1) {
        const int bit = x * kHold;
#pragma unroll
        for (int u = 0; u < x; ++u)
          m[u] = (lane & bit ? m[u + x] : m[u]) + __shfl_xor_sync(0xffffffffu, lane & bit ? m[u] : m[u + x], bit);
      }
      if (kHold == 2) m[0] += __shfl_xor_sync(0xffffffffu, m[0], 1);
      const float other = __shfl_xor_sync(0xffffffffu, m[0], 16);
      const float put0 = Job::DELTA ? beta * (v - m[0]) : beta * v;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float put = __shfl_sync(0xffffffffu, put0, u * kHold);
        z[u].x = fmaf(kk.x, put, z[u].x);
        z[u].y = fmaf(kk.y, put, z[u].y);
        z[u].z = fmaf(kk.z, put, z[u].z);
        z[u].w = fmaf(kk.w, put, z[u].w);
        if (on && c0 + u < a.dv) *reinterpret_cast<float4*>(S + u * a.dk) = z[u];
      }
      fence_async_smem();   // (the copy back reads what was written here)
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(done0 + 8 * s);
        mbar_arrive(taken0 + 8 * place);
      }
      o = fmaf(put0, kq, other);
    }
    if (Job::NORM) {
      const float part = warp_sum(has ? o * o : 0.f);
      if (lane == 0) red[n & 1][w] = part;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kStreamWarps) : "memory");
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < kStreamWarps; ++i) ss += red[n & 1][i];
      o *= (1.0f / sqrtf(ss / (float)a.dv + job.eps)) * ww;
    }
    if (has && alive) job.store(t, h, mine, o);
    ++n;
  }
}

// Whether states of these sizes go through the stream, and the launch.
static inline bool state_stream_fits(int dk, int dv, const void* state) {
  return dk % 4 == 0 && dk > 64 && dk <= kStreamDim && dv % 4 == 0 && dv > 32 && dv <= kStreamDim &&
         (reinterpret_cast<uintptr_t>(state) & 15) == 0;
}

template <class Job>
static int state_stream_launch(StateStream a, const Job& job, cudaStream_t stream) {
  const int bytes = a.dk * a.dv * 4;
  a.stages = kStreamBytes / bytes < kStreamStages ? kStreamBytes / bytes : kStreamStages;
  const long long items = (long long)a.n_entries * a.H;
  if (items > 0x3fffffffll) return CCB_REFUSE_SIZE;
  const int grid = (int)(items < 148 ? items : 148);
  static std::atomic<unsigned long long> done[2];
  const bool wide = a.dv > 64;
  const auto kernel = wide ? state_stream_kernel<Job, 16> : state_stream_kernel<Job, 8>;
  const int rc = ccb_allow_smem(kernel, kStreamBytes, done[wide]);
  if (rc != 0) return rc;
  ccb_launch_ex(true, kernel, dim3(grid), dim3(kStreamThreads), (size_t)a.stages * bytes, stream, a, job);
  return ccb_launch_status();
}

}  // namespace ccb
