// nav_engine.cuh -- one thread per track, the tracks of a block regrouped by the
// kind of volume they are in before every step.
//
// With a warp per track (navigation.cuh) every scalar part of a step, the frame
// changes, the mother's distances, the relocation, is executed by 32 lanes for one
// track, and the daughter loops fill the warp only where a volume has many
// daughters.  With a thread per track those parts serve 32 tracks at once, provided
// the tracks of a warp do the same thing: a track in a sensor (no daughters) and one
// in a module (a box with daughters) do not.  So a block keeps its tracks in shared
// memory and, before each step, sorts them by class (the mother's shape, with or
// without daughters; tracks still to be located are a class of their own): a
// counting sort over 32 classes, a few dozen instructions a track against the
// thousands of a step.  The tracks in wide volumes (hundreds of daughters) are the
// last class: each is stepped by a whole warp, which searches the daughters' boxes
// 32 at a time, so no thread holds its block up for a long list; the warps take these
// tracks one by one as they finish their threads' steps (a fixed share each kept the
// block waiting: traces of 65,536 detector tracks 3,226 us, now 3,102).  A finished
// track's slot takes the next track of the block's stream (grid-stride): the grid's cap
// of 1,184 blocks has 151,552 slots, so calls of more tracks than that refill, and in
// smaller ones a block thins out to its slowest track.
#pragma once
#include "navigation.cuh"

namespace vgb {

constexpr int kEngThreads = 128;  // and as many tracks a block
constexpr int kEngWarps = kEngThreads / 32;
constexpr int kEngBlocks = 4;  // resident blocks an SM: 128 registers a thread
constexpr int kEngClasses = 32;
constexpr int kEngEmpty = kEngClasses - 1;
constexpr int kEngWarp = kEngClasses - 2;  // tracks a whole warp steps
constexpr int kEngLocate = 0;
constexpr int32_t kLevelLocate = -1;  // NavTrack::path.level of a track to be located
static_assert(kEngClasses * kEngWarps == kEngThreads, "one counter a slot");
static_assert(kEngWarps <= 8, "WarpLanes::scratch");

// A track while its thread works on it.
struct NavTrack {
  V3<double> p, d;
  NavPath path;
  int32_t k;      // steps taken
  int32_t left;   // server requests only: steps left in this launch
  uint64_t hash;  // server requests only
};

// The tracks of a block.
struct NavPool {
  double c[6][kEngThreads];
  uint64_t hash[kEngThreads];
  int64_t idx[kEngThreads];
  int32_t k[kEngThreads];
  int32_t left[kEngThreads];
  int32_t level[kEngThreads];
  int32_t v[kNavMaxLevels][kEngThreads];
  int32_t count[kEngThreads];  // tracks per (class, warp), then their first places
  int32_t wsum[kEngWarps];
  int32_t next;  // the next track of the last class that a warp takes
  uint8_t boundary[kEngThreads];
  uint8_t key[kEngThreads];
  uint8_t order[kEngThreads];
};

VGB_D void pool_put(NavPool &S, int s, const NavTrack &t) {
  S.c[0][s] = t.p.x; S.c[1][s] = t.p.y; S.c[2][s] = t.p.z;
  S.c[3][s] = t.d.x; S.c[4][s] = t.d.y; S.c[5][s] = t.d.z;
  S.hash[s] = t.hash;
  S.k[s] = t.k;
  S.left[s] = t.left;
  S.level[s] = t.path.level;
  S.boundary[s] = t.path.boundary;
  for (int i = 0; i < t.path.level; ++i) S.v[i][s] = t.path.v[i];
}
VGB_D void pool_get(const NavPool &S, int s, NavTrack &t) {
  t.p = {S.c[0][s], S.c[1][s], S.c[2][s]};
  t.d = {S.c[3][s], S.c[4][s], S.c[5][s]};
  t.hash = S.hash[s];
  t.k = S.k[s];
  t.left = S.left[s];
  t.path.level = S.level[s];
  t.path.boundary = S.boundary[s];
  for (int i = 0; i < t.path.level; ++i) t.path.v[i] = S.v[i][s];
}
VGB_D uint8_t track_class(const NavGeom &G, const NavPath &p) {
  if (p.level <= 0) return kEngLocate;
  const NavVol v = nav_vol(G, p.top());
  if (v.wide != 0) return kEngWarp;
  return (uint8_t)(1 + 2 * (v.type - 1) + (v.dcount > 0 ? 1 : 0));
}
static_assert(1 + 2 * 13 < kEngWarp, "a class for every shape, with and without daughters");

// Sorts the block's slots by class into S.order; returns how many hold a track.
VGB_D int pool_sort(NavPool &S) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  __syncthreads();  // the last step's slots are written, its places read
  S.count[t] = 0;
  if (t == 0) S.next = 0;
  __syncthreads();
  const int key = S.key[t];
  const unsigned m = __match_any_sync(0xffffffffu, key);
  const int rank = __popc(m & ((1u << lane) - 1u));
  if (rank == 0) S.count[key * kEngWarps + w] = __popc(m);
  __syncthreads();
  const int v = S.count[t];
  int incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) S.wsum[w] = incl;
  __syncthreads();
  int base = 0;
  for (int i = 0; i < w; ++i) base += S.wsum[i];
  S.count[t] = base + incl - v;
  __syncthreads();
  S.order[S.count[key * kEngWarps + w] + rank] = (uint8_t)t;
  __syncthreads();
  return S.count[kEngEmpty * kEngWarps];
}

// Runs the tracks 0 .. n-1 of a client:
//   load(i, track)     -> the track, or false when there is nothing to do for it
//   step<L>(G, i, track) -> one locate or one step by L's lanes; false when the
//                         track is done (lane 0 has written its results)
template <class C>
VGB_D void nav_engine(const NavGeom &G, const C &client, int64_t n) {
  __shared__ NavPool S;
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * kEngThreads;
  // the first track from i on that has work, into a slot
  auto fill = [&](int slot, int64_t i, NavTrack &t) {
    uint8_t key = kEngEmpty;
    for (; i < n; i += stride) {
      if (client.load(i, t)) {
        S.idx[slot] = i;
        pool_put(S, slot, t);
        key = track_class(G, t.path);
        break;
      }
    }
    S.key[slot] = key;
  };
  auto after = [&](int slot, int64_t i, NavTrack &t, bool more) {
    if (more) {
      pool_put(S, slot, t);
      S.key[slot] = track_class(G, t.path);
    } else {
      fill(slot, i + stride, t);
    }
  };
  NavTrack t;
  fill(threadIdx.x, (int64_t)blockIdx.x * kEngThreads + threadIdx.x, t);
  for (;;) {
    const int live = pool_sort(S);
    if (live == 0) return;
    const int warp_first = S.count[kEngWarp * kEngWarps];  // first place of the last class
    if ((int)threadIdx.x < warp_first) {
      const int slot = S.order[threadIdx.x];
      const int64_t i = S.idx[slot];
      pool_get(S, slot, t);
      after(slot, i, t, client.template step<OneLane>(G, i, t));
    }
    __syncwarp();
    // the warps share the last class's tracks out as they get done
    for (;;) {
      int j = 0;
      if (lane == 0) j = warp_first + atomicAdd(&S.next, 1);
      j = __shfl_sync(0xffffffffu, j, 0);
      if (j >= live) break;
      const int slot = S.order[j];
      const int64_t i = S.idx[slot];
      pool_get(S, slot, t);
      const bool more = client.template step<WarpLanes>(G, i, t);
      __syncwarp();
      if (lane == 0) after(slot, i, t, more);
      __syncwarp();
    }
  }
}

// Whether a call of n tracks runs them by threads instead of by warps.  A warp
// finishes its track's step sooner (3 us against 25 in the layered detector), a
// thread's step costs a fifth of the instructions: few tracks go to warps, many to
// threads.  The lines lie where the two cross.  Measured (B200, us by warps / by
// threads): detector steps of 8,192 tracks 55 / 88, of 50,021 264 / 108; its traces
// of 64 steps of 16,384 tracks 1,807 / 1,950, of 65,536 7,756 / 3,102; ABBox traces of
// 16,384 2,501 / 3,674, of 32,768 5,349 / 4,135.  In mixed shapes a warp runs its
// daughters' different code one after the other, a class of threads walks one list:
// steps of 1,024 tracks 63 / 227, of 8,192 347 / 243, of 50,021 3,087 / 493; traces of
// 16,384 6,315 / 8,258, of 65,536 24,506 / 20,936; ABBox traces of 1,024 1,171 / 6,053,
// of 16,384 11,199 / 6,964.  LocatePoint of 12,288 points: detector 14.7 / 16.8, mixed
// shapes 35.1 / 35.1; of 16,384 17.6 / 18.9 and 43.3 / 35.2; of 24,576 21.9 / 18.8 and
// 59.6 / 36.6.
enum class NavCall { kLocate, kStep, kTrace, kAbboxStep, kAbboxTrace };
template <uint32_t kMask> bool nav_by_threads(NavCall call, int64_t n) {
  const bool mixed = kMask == kNavMaskAll;
  switch (call) {
    case NavCall::kLocate: return n >= 16384;
    case NavCall::kStep: return n >= (mixed ? 6144 : 16384);
    case NavCall::kTrace: return n >= (mixed ? 40960 : 20480);
    case NavCall::kAbboxStep: return n >= (mixed ? 5120 : 20480);
    case NavCall::kAbboxTrace: return n >= (mixed ? 10240 : 28672);
  }
  return false;
}

inline int engine_grid(int64_t n) {
  const int64_t want = (n + kEngThreads - 1) / kEngThreads;
  const int64_t cap = 148 * 8;
  return (int)(want < 1 ? 1 : (want > cap ? cap : want));
}

}  // namespace vgb
