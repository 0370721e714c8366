// pool.cuh -- the persistent photon-pool kernel.
//
// One CTA per SM slot stays resident for the whole run (the replacement of the reference's
// OpenMP team, cpp/3d/MC3D.hpp:1670-1700).  Every lane carries one photon; when photons
// end, the warp ballots its dead lanes and hands them the next indices from a warp-owned
// chunk of the global photon counter (one atomic per chunk), once refill_min lanes are
// idle or on every 8th iteration, so a warp never runs half-empty for long while photons
// remain.  A one-job launch on a small mesh stages the job's accumulators in shared memory
// (LaunchParams::dense) and adds them to the job's arrays when the CTA ends.  A photon index
// selects its job (batched launches), its Philox stream (key = job seed, counter = photon
// index) or its tape segment, and the walk advances one element step per loop iteration.
// Each loop iteration polls nothing but registers; the host cancel flag is read every 1024
// iterations.
#pragma once
#include "walk2d.cuh"

namespace vmc {

template <bool K> __device__ __forceinline__ void start_rng(PhiloxT<K> &rng, const JobDev &J, int64_t q) {
  rng.start(J.seed, J.stream, (uint64_t)(q + J.poffset));
}
__device__ __forceinline__ void start_rng(TapeRng &rng, const JobDev &J, int64_t q) {
  rng.start_tape(J.tape + J.tape_off[q], J.tape + J.tape_off[q + 1]);
}

// the job whose photon range [begin[j], begin[j + 1]) holds photon p
__device__ __forceinline__ int find_job(const int64_t *begin, int njobs, int64_t p) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (begin[mid] <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ---- the end of a launch ----
// Once the photons have been handed out, lanes die and are not replaced, yet a warp costs as
// much with one live lane as with most of them: on the 648k-tet phantom, whose longest walks
// take ten times the mean, half of a 1e6-photon launch ran in warps that were mostly empty.
// So the CTA's warps then meet every kPackEvery steps, and when the photons alive would fit
// three quarters of the warps that hold them they are moved together through shared memory, a
// few words of the state at a time.  They stay in two warps while there are more than three, and
// the last three get a warp each: two warps fill an SM's four schedulers with the FP64 forms' two
// CTAs, and a warp of one photon takes one branch.  (Full warps to the end, two, four and eight
// warps at the least: 9.6, 8.7, 8.8 and 10.1 ms at 1e4 photons on the phantom, 13.4, 13.4, 14.9
// and 17.4 at 1e5, in FP64 78, 78, 84 and 96; at 1e3 there 38.7, and 33.0 with the last three
// apart.)  A photon's arithmetic does not depend on the lane that
// carries it.  With the photons of small launches dealt to all SMs alike (below): 35.9 ->
// 29.6 ms for 1e6 photons on the phantom (32.1 without), 20.5 -> 13.4 at 1e5, 13-18 -> 9.6 at
// 1e4; FP64 571 -> 313 ms at 1e5.  Meeting every 64 to 512 steps measured alike there; every 64
// cost the 2D square and a 2D frequency-domain mesh, whose walks are short, 2-4 %, and the 2D
// tracking form does without (kPack).
constexpr unsigned kPackEvery = 512;
// the warp of a CTA that comes first, by the CTA's place on its SM
__device__ __forceinline__ int warp_turn(const LaunchParams &lp, int warps) {
  return (int)((long long)blockIdx.x * lp.ctas_per_sm / gridDim.x) % warps;
}
template <class Slot>  // uint2 or uint4: the words moved between two barriers
struct Packer {
  static constexpr int kWords = sizeof(Slot) / 4;
  Slot *buf;  // one per thread of the CTA
  int src;    // the thread whose photon this one takes, -1: none
  // to: the thread that takes this one's photon (-1: none to give)
  __device__ __forceinline__ Packer(Slot *b, int to) : buf(b) {
    int32_t *from = reinterpret_cast<int32_t *>(b);
    __syncthreads();
    from[threadIdx.x] = -1;
    __syncthreads();
    if (to >= 0) from[to] = (int)threadIdx.x;
    __syncthreads();
    src = from[threadIdx.x];
    __syncthreads();
  }
  template <class T> __device__ __forceinline__ static void get(const T &x, uint32_t *w) { memcpy(w, &x, sizeof(T)); }
  template <class T> __device__ __forceinline__ static void set(T &x, const uint32_t *w) { memcpy(&x, w, sizeof(T)); }
  // moves the values given (each of 4, 8 or 16 bytes)
  template <class... T> __device__ __forceinline__ void operator()(T &...x) const {
    constexpr int n = (int)((sizeof(T) + ...) / 4);
    uint32_t w[(n + kWords - 1) / kWords * kWords] = {};
    int at = 0;
    ((get(x, w + at), at += (int)sizeof(T) / 4), ...);
#pragma unroll
    for (int i = 0; i < n; i += kWords) {
      Slot v;
      memcpy(&v, w + i, sizeof(Slot));
      buf[threadIdx.x] = v;
      __syncthreads();
      if (src >= 0) v = buf[src];
      __syncthreads();
      memcpy(w + i, &v, sizeof(Slot));
    }
    at = 0;
    ((set(x, w + at), at += (int)sizeof(T) / 4), ...);
  }
};

// R::kOneJob: a launch of one job, whose descriptor (lp.job0) and Philox round keys are read
// from the kernel parameters (constant bank) rather than from global memory and registers.
// kTab: a launch of at most kSmemJobs jobs whose CTAs first copy the job table and its
// photon prefix into shared memory, so that the walk reads the descriptor of each lane's
// job there instead of from global memory (the table follows the dynamic shared memory's
// start; multi-job launches stage no accumulators).
template <class W, class R, bool kTab>
__global__ void __launch_bounds__(256, W::kMinBlocks) pool_kernel(const __grid_constant__ LaunchParams lp) {
  constexpr bool kOne = R::kOneJob;
  static_assert(!(kOne && kTab), "a one-job launch has no job table");
  W s;
  R rng;
  if constexpr (kOne) rng.rk = lp.rk;
  const JobDev *jobs = lp.jobs;
  const int64_t *job_begin = lp.job_begin;
  if constexpr (kTab) {
    JobDev *tab = reinterpret_cast<JobDev *>(vmc_smem);
    int64_t *tbeg = reinterpret_cast<int64_t *>(vmc_smem + sizeof(JobDev) * (size_t)lp.njobs);
    const int nw = lp.njobs * (int)(sizeof(JobDev) / sizeof(uint64_t));
    const uint64_t *src = reinterpret_cast<const uint64_t *>(lp.jobs);
    uint64_t *dst = reinterpret_cast<uint64_t *>(tab);
    for (int i = threadIdx.x; i < nw; i += blockDim.x) dst[i] = __ldg(src + i);
    for (int i = threadIdx.x; i <= lp.njobs; i += blockDim.x) tbeg[i] = __ldg(lp.job_begin + i);
    __syncthreads();
    jobs = tab;
    job_begin = tbeg;
  }
  const JobDev *J = kOne ? &lp.job0 : jobs;
  Stage stg{nullptr, nullptr, 0u};
  if constexpr (W::kStaged) {
    if (lp.stage_slots > 0) {
      stg.val = reinterpret_cast<double *>(vmc_smem);
      stg.tag = reinterpret_cast<int32_t *>(vmc_smem + sizeof(double) * lp.stage_slots);
      stg.mask = (uint32_t)lp.stage_slots - 1u;
      for (int i = threadIdx.x; i < lp.stage_slots; i += blockDim.x) {
        stg.tag[i] = -1;
        stg.val[i] = 0.0;
      }
      __syncthreads();
    }
  }
  s.stage = stg;
  if (lp.dense > 0) {  // the CTA's copy of the single job's accumulators starts at zero
    double *sm = reinterpret_cast<double *>(vmc_smem);
    for (int i = threadIdx.x; i < lp.dense; i += blockDim.x) sm[i] = 0.0;
    __syncthreads();
  }
  bool alive = false;
  uint32_t n_steps = 0, n_scat = 0, n_done = 0;
  const unsigned lane = threadIdx.x & 31u;
  long long chunk_next;  // this warp's next photon
  int chunk_left;        // photons it may still take, -1: every photon has been handed out
  {
    // A launch with fewer photons than lanes deals them out, lp.fill to a warp (0 otherwise):
    // first to the warps that come first in their CTA, one of each, and so on, so that every SM
    // gets as many; "first" turns with the CTA's place on its SM, so that those warps sit on
    // different schedulers.  All other photons come from the launch's counter.
    const int warps = blockDim.x >> 5;
    const int k = ((int)(threadIdx.x >> 5) + warps - warp_turn(lp, warps)) % warps;
    chunk_next = min(((long long)k * gridDim.x + blockIdx.x) * lp.fill, (long long)lp.total);
    chunk_left = (int)min((long long)lp.fill, (long long)lp.total - chunk_next);
  }
  __shared__ uint32_t pack_count[2][8];
  __shared__ volatile int launch_dry;  // a warp of the CTA has found every photon handed out
  if (W::kPack) {
    if (threadIdx.x == 0) launch_dry = 0;
    __syncthreads();
  }
  bool dry = false;  // the CTA's warps meet and pack from now on
  const unsigned lt_mask = (1u << lane) - 1u;
  const int32_t cap = (int32_t)min(lp.max_steps, (int64_t)INT32_MAX);
  for (unsigned it = 0;; ++it) {
    if ((it & 31u) == 0u) {
      if ((it & 1023u) == 0u) {  // the host's cancel flag (an L2 round trip), every 1024 steps
        if (*reinterpret_cast<volatile const int32_t *>(&lp.ctl->cancel)) {
          if (alive) n_steps += (uint32_t)s.nsteps;  // an unfinished walk's steps count in the launch's total
          alive = false;
          chunk_left = -1;
          if (W::kPack) launch_dry = 1;
        }
      }
      if (W::kPack && !dry && __shfl_sync(kFull, launch_dry, 0) != 0) {
        dry = true;
        it = 0;
      }
      if (W::kPack && dry) {
        if (it % kPackEvery == 0u) {
          // every warp of the CTA comes here, the same number of times
          const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
          uint32_t *count = pack_count[(it / kPackEvery) & 1u];
          const unsigned live = __ballot_sync(kFull, alive);
          if (lane == 0) count[warp] = (uint32_t)__popc(live) | (chunk_left > 0 ? 0x10000u : 0u);
          __syncthreads();
          int all = 0, before = 0, used = 0;
          bool pending = false;
          for (int k = 0; k < warps; k++) {
            const int c = (int)(count[k] & 0xffffu);
            pending |= count[k] > 0xffffu;
            before += k < warp ? c : 0;
            all += c;
            used += c > 0;
          }
          if (all == 0 && !pending) break;
          const int want = pack_warps(all, warps);
          if constexpr (W::kPack && !R::kReplay) {
            if (!pending && (used < want || 4 * want <= 3 * used)) {
              const int k = before + __popc(live & lt_mask);
              const int to = alive ? pack_thread(k, all, want, warp_turn(lp, warps), warps) : -1;
              auto slot = rng.take_slot();  // the lanes' stream slots are the buffer
              const Packer<decltype(slot)> pack(rng.slots(), to);
              s.move(pack);
              rng.template move<W::kBuffered>(pack, slot);
              if constexpr (!kOne) pack(J);
              rng.put_slot(slot);
              alive = pack.src >= 0;
            }
          }
        }
        if (chunk_left <= 0 && !__any_sync(kFull, alive)) {
          it |= kPackEvery - 1u;  // nothing to do until the next meeting
          continue;
        }
      }
    }
    // refill only when some lane is idle and photons are left (one vote in the common case)
    if (chunk_left >= 0 && __any_sync(kFull, !alive)) {
      unsigned need = __ballot_sync(kFull, !alive);
      // short walks: wait (at most 7 iterations) until enough lanes are idle to launch together
      if (__popc(need) < lp.refill_min && (it & 7u) != 0u) need = 0u;
      while (need) {
        if (chunk_left == 0) {
          unsigned long long base = 0;
          if (lane == 0) base = atomicAdd(&lp.ctl->next_photon, (unsigned long long)lp.chunk);
          chunk_next = (long long)__shfl_sync(kFull, base, 0) + lp.next0;
          if (chunk_next >= lp.total) {
            chunk_left = -1;
            if (W::kPack) launch_dry = 1;
            break;
          }
          chunk_left = (int)min((long long)lp.chunk, (long long)lp.total - chunk_next);
        }
        const int rank = __popc(need & lt_mask);
        if (((need >> lane) & 1u) && rank < chunk_left) {
          const long long p = chunk_next + rank;
          if constexpr (!kOne) J = jobs + (lp.njobs > 1 ? find_job(job_begin, lp.njobs, p) : 0);
          const long long q = p - J->pbegin;
          start_rng(rng, *J, q);
          s.launch(*J, rng, q);
          alive = true;
          if constexpr (W::kLaunchLoss) {
            if (s.lost_at_launch(*J)) { alive = false; n_done++; }
          }
        }
        const int taken = min(__popc(need), chunk_left);
        chunk_next += taken;
        chunk_left -= taken;
        need = __ballot_sync(kFull, !alive);
      }
    }
    if (!W::kPack && chunk_left < 0 && !__any_sync(kFull, alive)) break;
    // Events (W::kDefer): what a step ends in besides a scatter and a common crossing, the
    // boundary, an interface, roulette, takes as many instructions as several steps, and with a few
    // of 32 lanes at it a warp paid for it in nearly every step.  Lanes with an event wait until
    // they are a quarter of the warp's live ones.  1e6 photons on the 2D square, which meet one
    // every ten steps, 0.855 -> 0.705 ms (an eighth: 0.76, a third: 0.72), in FP64 5.8 -> 5.1;
    // uneven 2D mesh 2.35 -> 2.31 and 4.3 -> 3.9; a small tetrahedral box in FP64 7.0 -> 6.3.  The
    // FP32 tetrahedral walk, with one in a hundred steps, loses more by the waiting (1e7 photons on
    // the phantom 187 -> 220 ms, at a sixteenth 199) and does without; so would a mesh whose
    // index of refraction changes at every face (0.59 -> 0.65 ms; 0.70 before these forms).
    const auto ended = [&] {
      n_done++;
      n_steps += (uint32_t)s.nsteps;
      job_count_add(*J, kJcSteps, (unsigned long long)s.nsteps);
    };
    const auto step = [&] {
      if constexpr (W::kCap32) {
        alive = s.step(*J, rng, cap, n_scat);
      } else {
        const int r = s.step(*J, rng, lp.max_steps);
        n_scat += r == kScattered;
        alive = r <= kAliveMax;
      }
    };
    if constexpr (W::kDefer) {
      const bool was = alive;
      if (alive && !s.pending()) step();
      const bool event = alive && s.pending();
      const unsigned events = __ballot_sync(kFull, event);
      if (events && 4 * __popc(events) >= __popc(__ballot_sync(kFull, alive))) {
        if (event) alive = s.event(*J, rng, cap, n_scat);
      }
      if (was && !alive) ended();
    } else if (alive) {
      step();
      if (!alive) ended();
    }
  }
  if constexpr (W::kStaged) {
    // every warp of the CTA has left the loop: add the staged sums to the accumulator
    if (lp.stage_slots > 0) {
      __syncthreads();
      double *ER = lp.jobs[0].ER;
      for (int i = threadIdx.x; i < lp.stage_slots; i += blockDim.x) {
        const int32_t t = stg.tag[i];
        if (t >= 0 && stg.val[i] != 0.0) atomicAdd(ER + t, stg.val[i]);
      }
    }
  }
  if (lp.dense > 0) {
    // every warp of the CTA has left the loop: add the CTA's accumulators to the job's
    __syncthreads();
    const double *sm = reinterpret_cast<const double *>(vmc_smem);
    double *acc = kOne ? lp.job0.ER : lp.jobs[0].ER;
    for (int i = threadIdx.x; i < lp.dense; i += blockDim.x) {
      const double v = sm[i];
      if (v != 0.0) red_global(acc + i, v);
    }
  }
  unsigned long long a = n_steps, b = n_scat, c = n_done;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFull, a, o);
    b += __shfl_xor_sync(kFull, b, o);
    c += __shfl_xor_sync(kFull, c, o);
  }
  if (lane == 0) {
    atomicAdd(&lp.ctl->steps, a);
    atomicAdd(&lp.ctl->scatters, b);
    atomicAdd(&lp.ctl->done_photons, c);
  }
}

}  // namespace vmc
