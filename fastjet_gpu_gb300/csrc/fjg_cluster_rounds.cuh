// Clustering of one event per CTA in rounds of independent steps (sm_103a).
//
// The sequential algorithm takes one merge or promotion per step, the one with
// the smallest key.  What it does in one place of the rapidity-azimuth plane
// depends only on what happened within R of there, so steps far enough apart
// commute: their order decides the order of the output records, not what is
// merged.  This kernel fires many steps per round, each where it is the next
// one of its surroundings, checks that firing them early changed nothing, and
// sorts the records into the sequential order at the end.  A step-by-step
// kernel spends its time in latency (an FP64 kinematics chain, reductions,
// barriers); a round pays that once for all its steps.
//
// Sequential time.  The step E that merges c and j (or promotes c) with exact
// key k and label l (the winner's label; the lower one of mutual neighbours)
// has the time
//     T(E) = (k, l, 0)               if (k, l) > (M, m) of T(c) and T(j),
//            the larger of T(c), T(j) with its depth one higher   otherwise,
// where T(c) = (M, m, depth) is the time of the step that made c (before every
// time for an input particle).  In the sequential run the times of the steps
// increase: a step whose key is below an earlier one's became possible only
// with the step that made one of its pseudojets, and follows it directly.
// Conversely a set of steps sorted by T is the sequential run if, whenever two
// pseudojets x and y exist at the same time and E is the first step (in T) that
// takes either, then T(E) < T(x, y), the time the pair would have, and
// T(E) < the time of the promotion of the one it takes -- E being that pair or
// promotion excepted: the sequential run would otherwise have taken the pair or
// promotion first.  Two checks establish this; each compares in FP32 intervals
// and in FP64 where those cannot decide:
//   D1  when E fires: against every pseudojet within R of c and of j that
//       exists in the same round (before the round's steps are applied);
//   D2  when E makes a new jet a: against every pseudojet within R of a that a
//       step with a later time than T(E) has already taken.
// Two pseudojets that exist in the same round are covered by D1 of the first
// step that takes one of them, two that never do by D2 of the later one.
// T(x, y) >= d_xy, so with thr = k for the one whose own time sets a chained
// T(E) and thr = T(E)'s key part for the other, a pair is a conflict only if
// d_xy <= thr (an exact tie counts), d_xy is at most both weights and the other
// is not younger than E.  After a conflict the line of steps that came too
// early (round_line) and all that was fired since are taken back (round_undo), and
// its slots are held until the other step's time; where that is not enough, a wider
// range follows, and rounds of the one earliest step, which cannot conflict but for
// exact ties.  Those, and events with too many conflicts, are handed to the
// step-by-step kernel (retry list) and this kernel's work is dropped.  So the rule
// that picks the steps of a round only has to be good, not proven.
//
// Choice of a round's steps.  Tiles of side >= R/2; per tile the slot with the
// smallest (P, key), P being the FP32 lower bound of its step's time.  A tile
// whose minimum is the smallest of its 5x5 tiles is a candidate; it fires if
// no tile closer to c than 1.5 R and the distance of c and j (from the point to
// the tile) has an earlier minimum.  For kt and C/A, whose weights do not fall
// in a merge, it is R and shrinks to that of pairs with d below the candidate's P
// (48 kt events of 8000: 17.1 ms with 1.5 R, 16.0 with R; 600 events of 1500, 5.9
// and 5.4, C/A 7.6 and 7.1; with 0.7 R conflicts come: kt 21.2 and 15.2).  Steps a
// round on the benchmark's kind of events: anti-kt R = 0.4 4 at 200 particles, 10
// at 1500, 8 to 6 at 8000 to 40,000 dense ones, R = 0.8 3; with 1.5 R kt R =
// 0.6 12 at 1000, 14 at 20,000; C/A R = 0.8 8 at 1000.  Conflicts with a range of
// 1.5 R: none in 1100 events of up to 4000 particles (anti-kt R = 0.4, kt, C/A),
// in about 2 % of anti-kt R = 0.8 events of 3000 and in 2 to 8 % of dense anti-kt
// R = 0.4 events of 8000 to 15,000; those of 40,000 and more, where a hard jet's
// chain of steps reaches further, have one or several.  A conflict costs 30 to 900
// rounds (6000 to 10,000 dense particles), so events above 20,000 begin with 1.8 R: six
// batches of 64 events of 10,000 to 60,000 particles take 320 to 332 ms, 320 to 338 with
// 1.5 R, 304 to 373 with 1.65 R, 341 to 357 with 2.0 R.
//
// A round (F steps), eight warps or so:
//   A   candidates (a thread per tile); range test (eight lanes per candidate),
//       and the keys, times and thresholds of the steps that pass.
//   B   new jets' azimuth, rapidity and weight, and what takes the steps back:
//       four warps, a lane per step;
//       meanwhile the other warps go over the windows of c and j: D1, and the
//       slots whose neighbour is taken ("targets").
//   C   the new jets' state and the tile lists (a lane per step).
//   D   the new jets' windows (their neighbours; slots they are closer to), the
//       targets' searches, and D2 over the dead of the new jets' windows, by
//       groups of 8 or 32 lanes.
//   E   slots to which two new jets were closer: searched.
//   F   changed tiles: lists compacted, minima taken.
//
// Windows are the 5x5 tiles around a slot's tile; they hold everything within
// R (1 + 1e-4).  fjg_cluster_tiled.cuh proves that windowed neighbours select
// what the all-pairs rule selects.
#pragma once

#include <type_traits>

#include "fjg_cluster.cuh"

namespace fjg {

// Which events the rounds kernel takes.  Its gain is the number of steps a round
// holds, which falls with R^2 (the area a step keeps to itself), and a round
// costs about three steps of the step-by-step kernels.
//   One    a single event, in the widest CTA of either kernel.
//   Few    up to an SM per event, and Some, half an SM: the call lasts as long as
//          its slowest event, one with conflicts, or one left to the step-by-step
//          kernel after all, so the rounds have to win by more than in the mean.
//   Many   the SMs are shared, instructions count, of which a round's fixed part is
//          many for small events.
//   ServeOne, Serve   a server's micro-batch of one request, and of several: as One
//          and Few, but the step-by-step kernels run in the shapes with the most
//          events per second, and the rounds kernel with 128 to 512 threads.
// Measured on GB300, rounds / step by step (in its best shape but for the server),
// anti-kt unless noted.  One: 24 events, mean (worst).  Few and Some: calls of 20 to
// 300 events of a size, best to worst of the calls.  Serve: bursts of 16, 64 and 170
// requests of a size, the burst's time.
//   One    R 0.4: 160 0.98 (1.36), 200 0.85 (1.24), 256 0.69 (0.96), 1000 0.36;  R 0.6: 256 0.79 (1.04), 320 0.74 (0.94)
//          R 0.8: 512 0.92 (1.14), 1000 0.82 (0.98), 3000 0.88 (1.01);  R 1.0: 512 1.22, 2000 1.33
//          kt R 0.6: 200 0.72 (0.95), R 1.0: 320 0.64 (0.83), R 1.3: 600 0.77 (0.90), R 1.5: 700 0.92, 3000 1.03
//          C/A R 0.8: 160 0.80, R 1.2: 320 0.74 (0.93)
//   Few,   R 0.4: 200 1.15-1.38, 256 1.02-1.12 (Some: 1.04-1.26), 320 0.76-0.86, 1000 0.37-0.53;  R 0.5: 320 0.76-0.94
//   Some   (of 96 events of 17 to 301, few of them near the largest: rounds from 224 on 0.77 ms, from 257 on 0.83)
//          R 0.6: 320 0.89-1.06, 512 0.78-0.99, 600 0.68-0.82;  R 0.7: 600 0.83-0.95, 2000 0.77-0.89
//          R 0.8: 320 1.15-1.31, 1000 0.89-1.02, 3000 0.87-1.11
//          kt R 0.6: 256 0.84-1.03, 320 0.63-0.84, R 1.0: 320 0.82-1.09, 700 0.59-0.71, R 1.3: 600 0.87-0.99,
//          R 1.5: 700 1.04-1.17;  C/A R 0.8: 256 0.87-1.18, 320 0.71-0.92, R 1.2: 512 0.80-1.05, 700 0.72-0.88
//   Many   (ms) R 0.4: 2000 of 260-512 6.9 -> 6.3, 1000 of 600-1000 11.1 -> 5.9, 600 of 1100-2000 18.0 -> 6.9
//          R 0.6: 1000 of 600-1000 11.1 -> 9.3, 600 of 1100-2000 17.8 -> 17.9
//          kt R 0.6: 3000 of 150-256 4.7 -> 7.1, 1000 of 600-1000 9.8 -> 5.7
//          kt R 1.0: 1000 of 600-1000 9.9 -> 9.6, 600 of 1100-2000 17.8 -> 10.4;  C/A R 1.2: 10.1 -> 14.5, 18.3 -> 12.8
//   ServeOne  R 0.4: 112 0.87, 400 0.42;  R 0.8: 112 0.92, 1000 0.64, 4000 0.87;  R 1.0: 112 1.15, 1500 1.00
//          kt R 1.2: 112 0.84, 1000 0.55;  C/A R 1.2: 112 0.91, 1000 0.52
//   Serve  R 0.4: 200 1.48 1.22 1.12, 400 1.10 0.76 0.79, 512 1.01 0.62 0.79, 1000 0.62 0.43 0.73
//          R 0.5: 700 1.22 0.64 0.98, 1000 0.81 0.61 0.78, 1500 1.00 0.74 0.71;  R 0.6: 1500 1.16 0.90 0.87
//          kt R 0.6: 512 0.89 0.62 0.77;  R 1.0: 700 1.37 0.73 0.90, 1000 0.91 0.67 0.85, 1500 1.08 0.80 0.81
//          C/A R 0.8: 512 0.96 0.53 0.76, R 1.2: 1500 1.28 0.96 0.95
//   above 4096   alone / calls of 40 to 320:  R 0.4: 0.20-0.24 / 0.17-0.32;  R 0.8: 0.47-0.63 / 0.42-0.76
//                R 1.0: 0.64-0.83 (0.91) / 0.85-1.20;  R 1.05: 0.70-0.87 (0.97) / 0.91-1.05
//                kt R 1.5: 0.40-0.48 / 0.35-0.54, R 2.0: 0.54-0.64 / 0.50-0.70;  C/A R 2.0: 0.53-0.63 / 0.50-0.68
//                (ms) R 0.4: 12,000 123 -> 31, 58,000 700 -> 285, 250,000 6760 -> 3190;  R 0.6: 100,000 2350 -> 1610
enum { kRoundsNone = 0, kRoundsMany, kRoundsSome, kRoundsFew, kRoundsOne, kRoundsServe, kRoundsServeOne };

// In each mode the rule falls with R, and with n it changes at most once among the
// sizes of one list, from refusing to taking (the launchers count on it).
__host__ __device__ inline bool rounds_take(int mode, int n, int algo, double R) {
  if (mode == kRoundsNone) return false;
  const bool antikt = algo == -1, alone = mode == kRoundsOne || mode == kRoundsServeOne;
  if (n > 4096) return R <= (!antikt ? 2.0 : alone ? 1.05 : 0.85);
  switch (mode) {
    case kRoundsOne:
      if (antikt) return R <= 0.45 ? n >= 224 : R <= 0.65 ? n >= 320 : R <= 0.85 && n > 512;
      return R <= 0.8 ? n >= 200 : R <= 1.3 && n >= 320;
    case kRoundsFew:
      if (R <= (antikt ? 0.45 : 0.8)) return n >= 224;
      return R <= (antikt ? 0.55 : 1.0) ? n >= 320 : R <= (antikt ? 0.7 : 1.3) && n >= 600;
    case kRoundsSome: return R <= (antikt ? 0.55 : 0.8) ? n >= 320 : R <= (antikt ? 0.7 : 1.3) && n >= 600;
    case kRoundsServeOne: return R <= (antikt ? 0.85 : 1.2) && n >= 112;
    case kRoundsServe: return R <= (antikt ? 0.45 : 0.8) ? n > 512 : R <= (antikt ? 0.55 : 1.0) && n >= 1000;
    default:
      if (n <= 512) return n >= 400 && R <= (antikt ? 0.42 : 0.6);
      return R <= (antikt ? 0.55 : n <= 1024 ? 1.0 : 1.3);
  }
}

// The same for an event of a batch.  With one algorithm and R for all it is a
// comparison, and one thread of a CTA asks (next_event): the rule in line in every
// thread's event loop took a graph of 1024 events 5.38 -> 5.58 ms and a batch of 4096
// 17.5 -> 18.0.
static __device__ __noinline__ bool rounds_take_event(const BatchArgs* A, int e, int n) {
  return rounds_take(A->rounds_mode, n, A->algo ? A->algo[e] : A->algo_all, A->radius ? A->radius[e] : A->r_all);
}

__device__ __forceinline__ bool rounds_event(const BatchArgs& A, int e) {
  if (A.rounds_from == 0) return false;
  int64_t off;
  int n;
  event_range(A, e, off, n);
  return A.rounds_from > 0 ? n >= A.rounds_from : rounds_take_event(&A, e, n);
}

// The next event of the list that is for the rounds kernel, or for the others; -1:
// none is left (one thread of a CTA).
__device__ __forceinline__ int next_event(const BatchArgs& A, int count, bool rounds) {
#pragma unroll 1
  for (;;) {
    const int q = atomicAdd(A.queue, 1);
    if (q >= count) return -1;
    const int e = A.order[q];
    if (rounds_event(A, e) == rounds) return e;
  }
}

constexpr int kRoundSteps = 32;               // steps per round, at most (a lane each)
constexpr int kRoundBytesPerParticle = 384;   // workspace (368, and events start at whole sectors)
constexpr int kRoundMaxDirty = 384;
constexpr int kRoundMaxTargets = 128;
constexpr int kRoundSplit = 24;               // searches of a round, up to which several warps share each
constexpr int kRoundParts = 5;                // warps that share one, at most
constexpr int kRoundMaxCand = 704;            // 5x5 minima among 2048 tiles, also in one row
// range of the choice of steps, in units of R (see above): at first (anti-kt, its
// largest events, kt and C/A), and after a conflict
constexpr float kRoundReach = 1.5f, kRoundReachLarge = 1.8f, kRoundReachKt = 1.0f, kRoundReachWide = 2.25f;
constexpr int kRoundLargeFrom = 20000;
constexpr int kRoundCareRounds = 64;          // rounds that take care, more than twice those taken back
// Particles on a lattice (calorimeter towers) have many neighbours as far as another,
// whose steps' times tie in FP32: one conflict after the other.  An event in which
// more than one slot in kRoundTies has two such neighbours at first is left to the
// other kernels (events of free directions have none).  GB300, C/A R = 0.8, 0.087 x
// 0.087, step by step / in rounds until given up / left at once, ms: 1024 events of 700
// 13.2 / 20.0 / 14.2, of 1500 54.5 / 65.5 / 56.3; 100 of 700 4.5 / 6.2 / 3.9.  0.005 x 0.005,
// one in 300: 1024 of 1500 38.4 / 26.2 / -, kept.
constexpr int kRoundTies = 128;
constexpr int kRoundMaxBacks = 8;             // conflicts of an event, and one more per 2048 particles
constexpr int kRoundMaxTiles = 2048;
constexpr int kRoundMaxCells = 3072;          // with the frame
constexpr int kRoundFrame = 5;                // tiles around the grid: the range test's 1.5 R + R
constexpr int kRoundCrowded = 6;              // live slots per tile from which a search begins with the tiles around
constexpr int kRoundDense = 4;                // live slots per tile from which a warp reads lists together
constexpr int kRoundSmemMaxN = 4096;
constexpr int kRoundThreadsWs = 512;          // threads per event with its slots in the workspace
constexpr int kRoundSlotBytes = 36;           // shared memory per slot

// One step, stored at the slot it removes.
struct alignas(16) RoundRec {
  double M;   // its time: (M, l, depth)
  double d;   // recorded distance
  int l, depth;
  int a;      // merged into slot a, or -1 (promotion)
  int round;  // in which it was fired
};

struct RoundTime {
  double M;
  int l, depth;
};

__device__ __forceinline__ bool time_less(const RoundTime& x, const RoundTime& y) {
  if (x.M != y.M) return x.M < y.M;
  if (x.l != y.l) return x.l < y.l;
  return x.depth < y.depth;
}

constexpr unsigned kRoundNone = 0xffffffffu;  // a tile without slots (P as a bit pattern; P >= 0 orders as integer)

// A slot's state in the workspace, by sectors: what windows are scanned for, what
// a slot that gets a neighbour needs, the momentum, the rest.  (Separate arrays
// took a cache line for each of the 17 words that a step writes: phase C of a
// round took 14 kcycles at 50,000 particles.)
struct alignas(16) RoundSlot {
  float2 xy;   // rap32, phi32
  float2 key;  // lower bounds of the key, and of its step's time (P)
  float nhi;   // neighbour distance, upper bound
  int nn;      // neighbour field
  float wlo;   // weight, lower bound; negated: the upper bound is the next float up
  int tile;    // kNone: taken
  double2 pos;  // rapidity, azimuth
  double tm;    // birth time M
  int2 tl;      // birth time l, depth
  double p[4];
  double w;
  float tlo;  // birth time's M, rounded down
  int at;     // position in its tile's list
  int parent;  // (output) what the slot was merged into, or its jet
  float hold;  // a step of this slot with P from here on waits until all P are above it (0: none)
  int pad[2];
};

// What the step that removed a slot took: [0] c, [1] j.
struct alignas(16) RoundDead {
  float4 geo[2];  // rap32, phi32, wlo, threshold rounded up
  int4 grp[2];    // groups of the dead of one tile with the same M and l: next group (by descending
                  // M), its M rounded up (float), first member, l
  RoundRec rec;
  int next[2];    // next member
  int2 tl;        // slot a before the step, to take it back: as in RoundSlot
  double p[4], w, tm;
  double2 pos;
  int pad[4];
};
static_assert(sizeof(RoundSlot) == 128 && sizeof(RoundDead) == 192, "whole sectors");

// The event's state.  SM (events of up to kRoundSmemMaxN particles): what every
// round reads is in shared memory, 36 bytes a slot, so that two CTAs share an
// SM; what single slots need, the dead and the records are always in the
// workspace: RoundSlot[N], RoundDead[N], then (not SM) lxy and members.
template <bool SM>
struct RoundWs {
  using Idx = typename std::conditional<SM, unsigned short, int>::type;  // slots, tiles, list positions
  static constexpr int kRoom = SM ? 3 : 4;  // list entries per particle
  static constexpr int kNone = SM ? 0xffff : -1;
  // neighbour field: slot, or kNoSlot; a target of this round; the key is the pair distance
  static constexpr int kSlotMask = SM ? 0x1fff : 0x1ffffff, kNoSlot = kSlotMask;
  static constexpr int kTarget = SM ? 0x4000 : 0x20000000, kPair = SM ? 0x8000 : 0x40000000;
  RoundSlot* slots;
  RoundDead* dead;
  Idx* members;  // [kRoom * N]
  float2* lxy;   // [kRoom * N] coordinates in list order, read with consecutive lanes (not SM)
  float2 *sxy, *skey;  // (SM) the slots' state
  float *snhi, *swlo;
  Idx *snn, *stile, *sat;
  __device__ __forceinline__ float2& xy(int s) const { return SM ? sxy[s] : slots[s].xy; }
  __device__ __forceinline__ float2& key(int s) const { return SM ? skey[s] : slots[s].key; }
  __device__ __forceinline__ float& nhi(int s) const { return SM ? snhi[s] : slots[s].nhi; }
  __device__ __forceinline__ float& wlo(int s) const { return SM ? swlo[s] : slots[s].wlo; }
  __device__ __forceinline__ Idx& nn(int s) const { return pick(snn, slots[s].nn, s); }
  __device__ __forceinline__ Idx& tile(int s) const { return pick(stile, slots[s].tile, s); }
  __device__ __forceinline__ Idx& at(int s) const { return pick(sat, slots[s].at, s); }
  __device__ __forceinline__ double2& pos(int s) const { return slots[s].pos; }
  __device__ __forceinline__ double& tm(int s) const { return slots[s].tm; }
  __device__ __forceinline__ int2& tl(int s) const { return slots[s].tl; }
  __device__ __forceinline__ float& tlo(int s) const { return slots[s].tlo; }
  __device__ __forceinline__ double& p4(int q, int s) const { return slots[s].p[q]; }
  __device__ __forceinline__ double& w(int s) const { return slots[s].w; }
  // the dead: 2b and 2b+1, what the step that removed slot b took
  __device__ __forceinline__ float4& dgeo(int i) const { return dead[i >> 1].geo[i & 1]; }
  __device__ __forceinline__ int4& dgrp(int i) const { return dead[i >> 1].grp[i & 1]; }
  __device__ __forceinline__ int& dnext(int i) const { return dead[i >> 1].next[i & 1]; }
  __device__ __forceinline__ RoundRec& rec(int b) const { return dead[b].rec; }
  // coordinates of slot u, entry i of the lists
  __device__ __forceinline__ float2 entry(int u, int i) const { return SM ? sxy[u] : lxy[i]; }
  __device__ __forceinline__ void place(int i, int u, float2 g) const {
    members[i] = (Idx)u;
    if (!SM) lxy[i] = g;
  }
  __device__ __forceinline__ double dr2(int s, int t) const {
    const double2 a = pos(s), b = pos(t);
    return dr2_64(a.x, a.y, b.x, b.y);
  }

 private:
  __device__ static __forceinline__ unsigned short& pick(unsigned short* a, int&, int s) { return a[s]; }
  __device__ static __forceinline__ int& pick(int*, int& x, int) { return x; }
};

template <bool SM>
__device__ __forceinline__ RoundWs<SM> round_ws(unsigned char* base, unsigned char* smem, int N, int cap) {
  RoundWs<SM> W{};
  const int64_t n = N;
  W.slots = reinterpret_cast<RoundSlot*>(base);
  W.dead = reinterpret_cast<RoundDead*>(base + 128 * n);
  if (!SM) {
    W.lxy = reinterpret_cast<float2*>(base + 320 * n);
    W.members = reinterpret_cast<typename RoundWs<SM>::Idx*>(base + 352 * n);  // to 368 n
    return W;
  }
  W.sxy = reinterpret_cast<float2*>(smem);
  W.skey = W.sxy + cap;
  W.snhi = reinterpret_cast<float*>(W.skey + cap);
  W.swlo = W.snhi + cap;
  W.snn = reinterpret_cast<typename RoundWs<SM>::Idx*>(W.swlo + cap);
  W.stile = W.snn + cap;
  W.sat = W.stile + cap;
  W.members = W.sat + cap;
  return W;
}

__device__ __forceinline__ float round_wlo(float w) { return fabsf(w); }
__device__ __forceinline__ float round_whi(float w) {
  return __float_as_int(w) < 0 ? __int_as_float((__float_as_int(w) & 0x7fffffff) + 1) : w;
}
__device__ __forceinline__ float round_weight(double w) {
  const float lo = __double2float_rd(w);
  return __double2float_ru(w) == lo ? lo : -lo;
}

// Fixed part of a CTA's shared memory.
struct RoundShared {
  // the event, for the routines that stay out of line
  EventCtx X;
  unsigned char* ws;
  float r2hi;  // R^2 rounded up, a little more
  float far2;  // two slots whose FP32 coordinates are further apart (squared) are beyond R
  int tiles, cells, slots;  // room
  double rmin, inv_side_r, inv_side_phi;
  float rmin32, side_r, side_phi;
  int nrap, nphi, sh, nt, pw;  // tile (u, v) is u << sh | v; nt = nrap << sh
  int lut[16];                 // 2^16 / k, rounded up
  double red[3][24];
  int scan_tmp[24];
  int event, overflow;
  // conflict flags of a round's phases A, B and D: each is read after the
  // barrier that closes its phase and written again only a round later, so
  // every thread of the CTA takes the same way
  int conflict[3];
  int back;  // round to go back to
  // of the steps found to be too early: round and slot of the first, and the latest
  // time (M, rounded down) that they should have waited for
  unsigned long long early;
  int hold;
  int hopeless, alive, backs;
  int ties;  // searches with two neighbours as far
  // rounds before `care_until` take care: 1: the wide range; 2: one step, that
  // with the earliest time
  int care, care_until;
  unsigned p_min;
  float reach;
  int n_cand, n_fire, n_targets, n_dirty;
  int task[2];
  // the round's steps: c, j (-1: promotion), tile and list position of the
  // slots they remove and keep, tile of the new jet
  int c[kRoundSteps], j[kRoundSteps], l[kRoundSteps], depth[kRoundSteps];
  int2 tp_b[kRoundSteps], tp_a[kRoundSteps];
  int tile_c[kRoundSteps], tile_j[kRoundSteps];
  float2 xy_c[kRoundSteps], xy_j[kRoundSteps], wlo[kRoundSteps];  // (weights of c and of j)
  int new_u[kRoundSteps], new_v[kRoundSteps];
  double M[kRoundSteps], key[kRoundSteps], thr_c[kRoundSteps], thr_j[kRoundSteps];
  double phi[kRoundSteps], rap[kRoundSteps], w[kRoundSteps], p4[4][kRoundSteps];
  int targets[kRoundMaxTargets];
  int parts_done[kRoundSplit];  // searches shared by several warps
  unsigned short cand[kRoundMaxCand];  // tiles
  unsigned short dirty[kRoundMaxDirty];
  unsigned dirty_bits[kRoundMaxTiles / 32];
  // slots taken by a step of this round, and given a new neighbour (round_bit)
  unsigned taken[kRoundSmemMaxN / 32], claimed[kRoundSmemMaxN / 32];
};

// After it, `cells` minima of P with the grid's frame (kRoundFrame on each side;
// columns of the frame repeat the tiles across the azimuth seam, so that a
// neighbourhood is read without wrapping) and 5-tile row minima, then `tiles`
// entries of the per-tile arrays, then the slots, or (not SM) the parts
// of shared searches and a word per thread.
__host__ __device__ constexpr size_t round_tile_bytes(int tiles, int cells) {
  return ((size_t)cells * 12 + (size_t)tiles * 22 + 16 + 15) & ~size_t(15);
}
__host__ __device__ constexpr size_t round_tile_bytes_sm(int tiles, int cells) {
  return ((size_t)cells * 8 + (size_t)tiles * 16 + 16 + 15) & ~size_t(15);
}
__host__ __device__ constexpr size_t round_tiles_at() { return (sizeof(RoundShared) + 15) & ~size_t(15); }
template <bool SM>
__host__ __device__ constexpr size_t round_slots_at(int tiles, int cells) {
  return round_tiles_at() + (SM ? round_tile_bytes_sm(tiles, cells) : round_tile_bytes(tiles, cells));
}
template <bool SM>
__host__ __device__ constexpr size_t round_smem_bytes(int tiles, int cells, int slots) {
  return round_slots_at<SM>(tiles, cells) +
         (SM ? (size_t)slots * kRoundSlotBytes : sizeof(Cert) * kRoundSplit * kRoundParts + sizeof(int) * kRoundThreadsWs);
}

template <bool SM>
struct RoundCtx {
  using Idx = typename RoundWs<SM>::Idx;
  RoundShared* S;
  unsigned* tmin;  // [cells] smallest P of the tile's slots
  unsigned* row;   // [cells] smallest P of the five tiles around, in the row
  unsigned* near;  // [cells] smallest P of a step that takes a slot of the tile (SM: tmin)
  int* count;      // [nt]
  int* head;       // [nt] groups of the dead
  float* head_m;   // [nt] the first one's M (0: none)
  Idx* slot;       // [nt] the slot of the minimum
  unsigned short* beside;  // [nt] the tile of its partner, or its own (not SM)
  Idx* start;      // [nt + 1]
  Cert* part;      // [kRoundSplit * kRoundParts] (not SM)
  int* shift;      // [threads] for_tiles (not SM)
  RoundWs<SM> W;
};

// The context, from shared memory (the per-slot pointers need the event set).
template <bool SM>
__device__ __forceinline__ RoundCtx<SM> round_ctx() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RoundCtx<SM> C;
  C.S = reinterpret_cast<RoundShared*>(smem_raw);
  const int tiles = C.S->tiles, cells = C.S->cells;
  C.tmin = reinterpret_cast<unsigned*>(smem_raw + round_tiles_at());
  C.row = C.tmin + cells;
  C.near = SM ? C.tmin : C.row + cells;
  C.count = reinterpret_cast<int*>(C.row + (SM ? cells : 2 * cells));
  C.head = C.count + tiles;
  C.head_m = reinterpret_cast<float*>(C.head + tiles);
  C.slot = reinterpret_cast<typename RoundCtx<SM>::Idx*>(C.head_m + tiles);
  C.start = C.slot + tiles;
  C.beside = reinterpret_cast<unsigned short*>(C.start + tiles + 2);
  C.part = reinterpret_cast<Cert*>(smem_raw + round_slots_at<SM>(tiles, cells));
  C.shift = reinterpret_cast<int*>(C.part + kRoundSplit * kRoundParts);
  C.W = round_ws<SM>(C.S->ws, smem_raw + round_slots_at<SM>(tiles, cells), C.S->X.N, C.S->slots);
  return C;
}

__device__ __forceinline__ int round_u(const RoundShared& S, double rap) {
  const int u = (int)floor((rap - S.rmin) * S.inv_side_r);
  return u < 0 ? 0 : (u >= S.nrap ? S.nrap - 1 : u);
}

__device__ __forceinline__ int round_v(const RoundShared& S, double phi) {
  const int v = (int)floor(phi * S.inv_side_phi);
  return v < 0 ? 0 : (v >= S.nphi ? S.nphi - 1 : v);
}

// What this kernel leaves to the step-by-step kernels.  A weight of 0 (kt without
// pT: a pair distance of 0 at any distance) or one that overflowed; a rapidity that
// did (no pT and E < |pz| gives +-infinity, sums beyond 1e154 NaN), or whose FP32
// distances could: a NaN bound certifies no neighbour, and the FP64 search that
// follows would find none within it.  Below 1e30 bounds may be infinite, never NaN.
__device__ __forceinline__ bool round_refuses(double w) { return !(w > 0.0 && w <= 1.7976931348623157e308); }
__device__ __forceinline__ bool round_refuses_rap(double rap) { return !(fabs(rap) < 1e30); }

// S.far2 for an event with |rapidity| up to rmax.  An FP32 coordinate is off by
// 2^-24 of itself (a rapidity of 1e5, of a particle on the beam line, by 0.004),
// so two slots within R can be 2^-23 (rmax + 4 pi) further apart in FP32; twice
// that, and 1e-3 and 1e-6 for the rounding of the distance and of the tiles' edges.
__device__ __forceinline__ float round_far2(float r2hi, double rmax) {
  const double d = sqrt((double)r2hi) + 0x1p-22 * (rmax + 12.6);
  return __double2float_ru(d * d * 1.001 + 1e-6);
}

// A box of tiles: nu rows from u0, nv columns from v0 (wrapping; nv <= 9).
struct RoundBox {
  int u0, nu, v0, nv;
};

// The smallest box holding the windows (5x5 tiles) of tiles t1 and t2, which
// lie within each other's.
__device__ __forceinline__ RoundBox round_box(const RoundShared& S, int t1, int t2) {
  const int u1 = t1 >> S.sh, v1 = t1 & ((1 << S.sh) - 1);
  const int u2 = t2 >> S.sh, v2 = t2 & ((1 << S.sh) - 1);
  RoundBox b;
  b.u0 = max(min(u1, u2) - 2, 0);
  b.nu = min(max(u1, u2) + 2, S.nrap - 1) - b.u0 + 1;
  int dv = v2 - v1;
  if (2 * dv > S.nphi) dv -= S.nphi;
  if (2 * dv < -S.nphi) dv += S.nphi;
  b.nv = 5 + abs(dv);
  b.v0 = v1 - 2 + min(dv, 0);
  if (b.v0 < 0) b.v0 += S.nphi;
  if (b.nv >= S.nphi) {
    b.v0 = 0;
    b.nv = S.nphi;
  }
  return b;
}

// Tile k of a box.
__device__ __forceinline__ int box_tile(const RoundShared& S, const RoundBox& b, int k) {
  const int du = (k * S.lut[b.nv]) >> 16;
  int v = b.v0 + (k - du * b.nv);
  if (v >= S.nphi) v -= S.nphi;
  return ((b.u0 + du) << S.sh) + v;
}

// Squared distance of a point to tile (u, v); the outermost rows hold what lies
// beyond them.
__device__ __forceinline__ float tile_d2(const RoundShared& S, float2 g, int u, int v) {
  const float lo = S.rmin32 + u * S.side_r;
  float dr = 0.0f;
  if (u > 0) dr = fmaxf(dr, lo - g.x);
  if (u < S.nrap - 1) dr = fmaxf(dr, g.x - lo - S.side_r);
  float dp = fabsf(g.y - (v + 0.5f) * S.side_phi);
  dp = fmaxf(fminf(dp, kTwoPiF - dp) - 0.5f * S.side_phi, 0.0f);
  return dr * dr + dp * dp;
}

// fn(slot, load(slot, coordinates)) for every list entry of the box's tiles k0 ..
// n-1 (the functions hold no warp collectives).  Lists in shared memory: a group
// of G lanes (8 or 32, the same in the whole warp), a lane per tile, two members
// at a time.  Lists in the workspace: a warp; a lane per tile first, which leaves
// out the tiles further than R from p and from q and adds the lengths up; then the lists as one sequence, every lane an
// entry of it, three at a time so that their loads are in flight together.
// (Lanes given to tiles, 32 / length tiles at a time, ran four times the
// instructions: lists differ in length.)  Lengths are bounded by the tile's room.
template <bool SM, class Load, class Fn>
__device__ __forceinline__ void for_tiles(const RoundCtx<SM>& C, const RoundBox& b, int k0, int n, int G, float2 p,
                                          float2 q, Load load, Fn fn) {
  const RoundShared& S = *C.S;
  constexpr int kNone = RoundWs<SM>::kNone;
  if (!SM) {
    constexpr int B = 3;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1, upto = below | (1u << lane);
    const float far2 = S.far2;
    int* shift = C.shift + (threadIdx.x & ~31);
#pragma unroll 1
    for (; k0 < n; k0 += 32) {
      const int k = k0 + lane, t = box_tile(S, b, k < n ? k : k0), st = C.start[t];
      const int u = t >> S.sh, v = t & ((1 << S.sh) - 1);
      int ln = 0;
      if (k < n && fminf(tile_d2(S, p, u, v), tile_d2(S, q, u, v)) <= far2)
        ln = min(C.count[t], (int)C.start[t + 1] - st);
      int end = ln;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(kFull, end, o);
        if (lane >= o) end += x;
      }
      const int total = __shfl_sync(kFull, end, 31), begin = end - ln;
      const unsigned some = __ballot_sync(kFull, ln > 0);
      if (ln > 0) shift[__popc(some & below)] = st - begin;
      __syncwarp();
      int before = -1;  // lists that begin before this point of the sequence
#pragma unroll 1
      for (int base = 0; base < total; base += 32 * B) {
        int u[B];
        float2 g[B];
        decltype(load(0, make_float2(0.0f, 0.0f))) d[B];
#pragma unroll
        for (int c = 0; c < B; ++c) {
          const unsigned at = (unsigned)(begin - base - 32 * c);
          const unsigned starts = __reduce_or_sync(kFull, ln > 0 && at < 32u ? 1u << at : 0u);
          const int i = base + 32 * c + lane, r = before + __popc(starts & upto);
          before += __popc(starts);
          const int e = i < total ? shift[r] + i : 0;
          u[c] = i < total ? (int)C.W.members[e] : kNone;
          g[c] = C.W.lxy[e];
        }
#pragma unroll
        for (int c = 0; c < B; ++c) d[c] = load(u[c] != kNone ? u[c] : 0, g[c]);
#pragma unroll
        for (int c = 0; c < B; ++c)
          if (u[c] != kNone) fn(u[c], d[c]);
        __syncwarp();
      }
    }
  } else {
#pragma unroll 1
    for (int k = k0 + (threadIdx.x & (G - 1)); k < n; k += G) {
      const int t = box_tile(S, b, k);
      const int st = C.start[t], m = min(C.count[t], (int)C.start[t + 1] - st);
#pragma unroll 1
      for (int i = 0; i < m; i += 2) {
        const int u0 = C.W.members[st + i], u1 = i + 1 < m ? (int)C.W.members[st + i + 1] : kNone;
        const int v0 = u0 != kNone ? u0 : 0, v1 = u1 != kNone ? u1 : v0;
        const auto d0 = load(v0, C.W.xy(v0)), d1 = load(v1, C.W.xy(v1));
        if (u0 != kNone) fn(u0, d0);
        if (u1 != kNone) fn(u1, d1);
      }
    }
  }
  __syncwarp();
}

template <bool SM, class Load, class Fn>
__device__ __forceinline__ void for_box(const RoundCtx<SM>& C, const RoundBox& b, int G, float2 p, Load load, Fn fn) {
  for_tiles(C, b, 0, b.nu * b.nv, G, p, p, load, fn);
}

// Combination of certificates over groups of G lanes (all lanes call).
__device__ __forceinline__ Cert cert_group(Cert c, int G) {
  if (G == 32) return cert_warp(c);
#pragma unroll 1
  for (int o = G / 2; o; o >>= 1) {
    Cert y;
    y.m1 = __shfl_xor_sync(kFull, c.m1, o);
    y.i1 = __shfl_xor_sync(kFull, c.i1, o);
    y.u1 = __shfl_xor_sync(kFull, c.u1, o);
    y.m2 = __shfl_xor_sync(kFull, c.m2, o);
    if (y.m1 < c.m1 || (y.m1 == c.m1 && (unsigned)y.i1 < (unsigned)c.i1)) {
      y.m2 = fminf(y.m2, c.m1);
      c = y;
    } else {
      c.m2 = fminf(c.m2, y.m1);
    }
  }
  return c;
}

__device__ __forceinline__ void round_dirty(RoundShared& S, int t) {
  const unsigned bit = 1u << (t & 31);
  if (!(atomicOr(&S.dirty_bits[t >> 5], bit) & bit)) {
    const int k = atomicAdd(&S.n_dirty, 1);
    if (k < kRoundMaxDirty) S.dirty[k] = (unsigned short)t;
  }
}

__device__ __forceinline__ void round_target(RoundShared& S, int t) {
  const int k = atomicAdd(&S.n_targets, 1);
  if (k < kRoundMaxTargets) S.targets[k] = t;
}

// A slot's bit of S.taken and S.claimed: its own, or (not SM) one of 4096 by a
// hash.  A bit shared with another slot costs time, not correctness: a step waits
// for the next round, a slot is searched.
template <bool SM>
__device__ __forceinline__ int round_bit(int s) {
  return SM ? s : (int)(((unsigned)s * 2654435761u) >> 20);
}

// True for the first caller of a round.
__device__ __forceinline__ bool round_first(unsigned* bits, int b) {
  const unsigned bit = 1u << (b & 31);
  return !(atomicOr(bits + (b >> 5), bit) & bit);
}

// The routines that a round's lanes call for single slots stay out of line: the
// kernel's straight-line code would not fit the instruction caches otherwise
// (400 KB inlined; a round took 1.5 to 2 times as long).

// Slot t's neighbour nn with distance interval [lo, hi]: neighbour, key and P;
// the tile is marked as changed.  The FP32 filter's interval is wide for close
// pairs (its bound is absolute), which FP64 settles, so that keys compare well:
// a neighbour's interval is narrower than 2^-16 of it.  Beyond R there is no
// neighbour: the lighter of such a pair is promoted before the pair's turn, and
// all that have c as their neighbour are found within R of c.  `keep`: kTarget, if the
// other groups of this phase are to leave t alone.  What may be needed is
// loaded at once.
template <bool SM>
__device__ __noinline__ void round_set(int t, int nn, float lo, float hi, int keep) {
  using Ws_ = RoundWs<SM>;
  const RoundCtx<SM> C = round_ctx<SM>();
  const EventCtx& X = C.S->X;
  const int n = nn < 0 ? t : nn;
  const float w = C.W.wlo(t), tlo = C.W.tlo(t), wn = C.W.wlo(n), tn = C.W.tlo(n);
  const double2 pt = C.W.pos(t), pn = C.W.pos(n);
  round_dirty(*C.S, C.W.tile(t));
  float klo = round_wlo(w), p = fmaxf(klo, tlo);
  int field = Ws_::kNoSlot;
  if (nn >= 0 && hi - lo > lo * 0x1p-16f) {
    const double d = dr2_64(pt.x, pt.y, pn.x, pn.y);
    lo = __double2float_rd(d);
    hi = __double2float_ru(d);
  }
  if (nn < 0 || lo > C.S->r2hi) {
    hi = C.S->r2hi;
  } else {
    float khi;
    int kind = key_interval(klo, round_whi(w), round_wlo(wn), round_whi(wn), lo, hi, X.ilo, X.ihi, klo, khi);
    if (kind < 0) {
      const double w64 = C.W.w(t);
      const double dp = pair_distance(w64, C.W.w(nn), dr2_64(pt.x, pt.y, pn.x, pn.y), X.inv_r2);
      kind = dp < w64 ? 1 : 0;
      klo = __double2float_rd(kind ? dp : w64);
    }
    p = fmaxf(klo, tlo);
    if (kind) p = fmaxf(p, tn);
    field = nn | (kind ? Ws_::kPair : 0);
  }
  C.W.key(t) = make_float2(klo, p);
  C.W.nhi(t) = hi;
  C.W.nn(t) = (typename Ws_::Idx)(field | keep);
}

// Slot t's neighbour by the exact minimum (dR2, label) over its window (whole
// warp), among those whose FP32 lower bound does not exceed u1.  Counts in S.ties if
// the second one is as far, in FP32.
template <bool SM>
__device__ __noinline__ int round_exact(int t, float u1) {
  const RoundCtx<SM> C = round_ctx<SM>();
  const int tile = C.W.tile(t);
  const RoundBox b = round_box(*C.S, tile, tile);
  const float2 gt = C.W.xy(t);
  const Bound bd = C.S->X.bd;
  unsigned long long bk = ~0ull, b2 = ~0ull;
  int bi = 0x7fffffff;
  for_box(C, b, 32, gt, [&](int, float2 g) { return g; },
          [&](int u, float2 gu) {
            float l, h;
            dr2_32(gt.x, gt.y, gu.x, gu.y, bd, l, h);
            if (u == t || l > u1) return;
            const unsigned long long k = dbits(C.W.dr2(t, u));
            if (arg_less(k, u, bk, bi)) {
              b2 = bk;
              bk = k;
              bi = u;
            } else if (k < b2) {
              b2 = k;
            }
          });
  const Arg r = arg_warp(bk, bi, bi);
  const double best = __longlong_as_double((long long)r.key);
  const double next = __longlong_as_double((long long)(bi == r.idx ? b2 : bk));  // (~0: a NaN)
  if (__any_sync(kFull, next - best <= best * 0x1p-22) && (threadIdx.x & 31) == 0) atomicAdd(&C.S->ties, 1);
  return r.idx;
}

// Stores slot t's neighbour from its group's certificate (every lane calls;
// lane `first` of the group holds the work, have: it has some).
template <bool SM>
__device__ __forceinline__ void round_settle(bool have, bool first, int t, const Cert& c, int keep) {
  const bool exact = have && first && c.i1 >= 0 && !cert_ok(c);
  unsigned todo = __ballot_sync(kFull, exact);
  if (have && first && !exact) round_set<SM>(t, c.i1, c.m1, c.u1, keep);
  __syncwarp();
  while (todo) {
    const int q = __ffs(todo) - 1;
    todo &= todo - 1;
    const int tq = __shfl_sync(kFull, t, q);
    const int nn = round_exact<SM>(tq, __shfl_sync(kFull, c.u1, q));
    // (an empty interval: the FP64 value is taken)
    if ((threadIdx.x & 31) == q) round_set<SM>(tq, nn, 0.0f, __int_as_float(0x7f800000), keep);
    __syncwarp();
  }
}

// The certificate of search `item` from its parts, each done by a warp (parts >
// 1; every lane calls): true for the last one, which holds the whole.
template <bool SM>
__device__ __forceinline__ bool round_join(const RoundCtx<SM>& C, Cert& c, int item, int part, int parts) {
  Cert* all = C.part + item * kRoundParts;
  const int lane = threadIdx.x & 31;
  int done = 0;
  if (lane == 0) {
    all[part] = c;
    __threadfence_block();
    done = atomicAdd(&C.S->parts_done[item], 1);
  }
  if (__shfl_sync(kFull, done, 0) != parts - 1) return false;
  __threadfence_block();
  c = cert_warp(lane < parts ? all[lane] : cert_empty());
  return true;
}

// Slot t's neighbour in its window, and its key (groups of G lanes; or one of
// several warps of search `item`; parts = 0: the tiles around first).
template <bool SM>
__device__ __noinline__ void round_search(bool have, int t, int G, int item, int part, int parts) {
  const RoundCtx<SM> C = round_ctx<SM>();
  const int tile = have ? (int)C.W.tile(t) : 0;
  RoundBox b = round_box(*C.S, tile, tile);
  if (!have) b.nu = 0;
  const float2 gt = C.W.xy(t);
  const Bound bd = C.S->X.bd;
  Cert x = cert_empty();
  bool near = false;
  if (!SM && parts == 0) {
    // many slots per tile: the tiles next to its own, beyond which all is further
    // than the smaller side
    if (have) {
      const int u = tile >> C.S->sh, v = tile & ((1 << C.S->sh) - 1);
      b.u0 = max(u - 1, 0);
      b.nu = min(u + 1, C.S->nrap - 1) - b.u0 + 1;
      b.v0 = v ? v - 1 : C.S->nphi - 1;
      b.nv = 3;
    }
    near = true;
    parts = 1;
  }
#pragma unroll 1
  for (;;) {
    const int nb = b.nu * b.nv;
    for_tiles(C, b, nb * part / parts, nb * (part + 1) / parts, G, gt, gt, [&](int, float2 g) { return g; },
            [&](int u, float2 gu) {
              float lo, hi;
              dr2_32(gt.x, gt.y, gu.x, gu.y, bd, lo, hi);
              if (u != t) cert_add(x, lo, hi, u);
            });
    x = cert_group(x, G);
    if (!near) break;
    near = false;
    const float side = fminf(C.S->side_r, C.S->side_phi) * 0.999f;
    if (!have || (x.i1 >= 0 && x.u1 <= side * side)) break;
    x = cert_empty();
    b = round_box(*C.S, tile, tile);
  }
  if (parts > 1 && !round_join(C, x, item, part, parts)) return;
  round_settle<SM>(have, (threadIdx.x & (G - 1)) == 0, t, x, RoundWs<SM>::kTarget);
}

// New jet a, with FP32 distance interval [lo, hi] to slot y (no target), may be
// closer to y than its neighbour.  Another jet may be given to y at the same
// time: whichever of y's words are seen, what is kept is closer than before,
// and of two that claim y the second has it searched.
template <bool SM>
__device__ __noinline__ void round_offer(int y, int a, float lo, float hi, float nhi) {
  using Ws_ = RoundWs<SM>;
  const RoundCtx<SM> C = round_ctx<SM>();
  if (!(hi < nhi * (1.0f - 0x1p-14f))) {
    const int cn = *(volatile typename Ws_::Idx*)&C.W.nn(y) & Ws_::kSlotMask;
    if (cn != Ws_::kNoSlot) {
      const double da = C.W.dr2(y, a), dc = C.W.dr2(y, cn);
      if (!(da < dc || (da == dc && a < cn))) return;
    }
  }
  if (round_first(C.S->claimed, round_bit<SM>(y)))
    round_set<SM>(y, a, lo, hi, 0);
  else
    round_target(*C.S, y);  // (phase E)
}

// D1 in FP64 (see the header): pseudojet x of a step with time part M and
// threshold thr against slot y.
template <bool SM>
__device__ __noinline__ bool round_d1_exact(int x, int y, double thr, double M) {
  const RoundCtx<SM> C = round_ctx<SM>();
  const EventCtx& X = C.S->X;
  const double wx = C.W.w(x), wy = C.W.w(y), ty = C.W.tm(y);
  const double d = pair_distance(wx, wy, C.W.dr2(x, y), X.inv_r2);
  return d <= thr && d <= fmin(wx, wy) && !(ty > M);
}

// The minimum of tile t (slot: P, neighbour field) into its cell and the frame's
// copies of it.
template <bool SM>
__device__ __forceinline__ void round_store_min(const RoundCtx<SM>& C, int t, unsigned p, int slot, int nn) {
  const RoundShared& S = *C.S;
  const int u = t >> S.sh, v = t & ((1 << S.sh) - 1);
  unsigned* row = C.tmin + (u + kRoundFrame) * S.pw + kRoundFrame;
  C.slot[t] = (typename RoundCtx<SM>::Idx)slot;
  if (!SM) {
    int beside = t;
    if (slot >= 0 && (nn & RoundWs<SM>::kPair)) beside = C.W.tile(nn & RoundWs<SM>::kSlotMask);
    C.beside[t] = (unsigned short)beside;
  }
  row[v] = p;
#pragma unroll 1
  for (int w = v - S.nphi; w >= -kRoundFrame; w -= S.nphi) row[w] = p;
#pragma unroll 1
  for (int w = v + S.nphi; w < S.nphi + kRoundFrame; w += S.nphi) row[w] = p;
}

__device__ __forceinline__ bool round_before(float2 x, int sx, float2 y, int sy) {
  return sy < 0 || x.y < y.y || (x.y == y.y && (x.x < y.x || (x.x == y.x && sx < sy)));
}

// Tile t's list compacted and its minimum (P, key, slot): a whole warp, or one
// thread.
template <bool SM>
__device__ __noinline__ void round_summary_warp(int t) {
  const RoundCtx<SM> C = round_ctx<SM>();
  using Idx = typename RoundWs<SM>::Idx;
  constexpr int kNone = RoundWs<SM>::kNone;
  if ((t & ((1 << C.S->sh) - 1)) >= C.S->nphi) return;
  const int lane = threadIdx.x & 31;
  const int st = C.start[t], m = min(C.count[t], (int)C.start[t + 1] - st);
  float2 best = make_float2(0.0f, 0.0f);
  int slot = -1, nn = 0, out = 0;
#pragma unroll 1
  for (int i0 = 0; i0 < m; i0 += 32) {
    const int i = i0 + lane;
    const int u = i < m ? (int)C.W.members[st + i] : kNone;
    const float2 gu = i < m ? C.W.entry(0, st + i) : make_float2(0.0f, 0.0f);
    const unsigned ball = __ballot_sync(kFull, u != kNone);
    if (u != kNone) {
      const int p = out + __popc(ball & ((1u << lane) - 1));
      if (p != i) {
        C.W.place(st + p, u, gu);
        C.W.at(u) = (Idx)p;
      }
      const float2 k = C.W.key(u);
      const int f = C.W.nn(u);
      if (round_before(k, u, best, slot)) {
        best = k;
        slot = u;
        nn = f;
      }
    }
    out += __popc(ball);
    __syncwarp();
  }
  const unsigned p = slot >= 0 ? __float_as_uint(best.y) : kRoundNone;
  const unsigned pb = __reduce_min_sync(kFull, p);
  const unsigned k = slot >= 0 && p == pb ? __float_as_uint(best.x) : kRoundNone;
  const unsigned kb = __reduce_min_sync(kFull, k);
  const unsigned sb = __reduce_min_sync(kFull, slot >= 0 && p == pb && k == kb ? (unsigned)slot : kRoundNone);
  const unsigned win = __ballot_sync(kFull, slot >= 0 && (unsigned)slot == sb);
  if (lane == (win ? __ffs(win) - 1 : 0)) {
    round_store_min(C, t, pb, (int)sb, nn);
    C.count[t] = out;
  }
}

template <bool SM>
__device__ __noinline__ void round_summary_thread(int t) {
  const RoundCtx<SM> C = round_ctx<SM>();
  using Idx = typename RoundWs<SM>::Idx;
  if ((t & ((1 << C.S->sh) - 1)) >= C.S->nphi) return;
  const int st = C.start[t], m = min(C.count[t], (int)C.start[t + 1] - st);
  float2 best = make_float2(0.0f, 0.0f);
  int slot = -1, out = 0;
#pragma unroll 1
  for (int i = 0; i < m; ++i) {
    const int u = C.W.members[st + i];
    if (u == RoundWs<SM>::kNone) continue;
    if (out != i) {
      C.W.place(st + out, u, C.W.entry(0, st + i));
      C.W.at(u) = (Idx)out;
    }
    ++out;
    const float2 k = C.W.key(u);
    if (round_before(k, u, best, slot)) {
      best = k;
      slot = u;
    }
  }
  round_store_min(C, t, slot >= 0 ? __float_as_uint(best.y) : kRoundNone, slot, slot >= 0 ? (int)C.W.nn(slot) : 0);
  C.count[t] = out;
}

// Tile lists from the live slots (whole CTA).  What the list area spares is
// spread over the lists as room for more.
template <bool SM>
__device__ __noinline__ void round_lists(int n) {
  const RoundCtx<SM> C = round_ctx<SM>();
  RoundShared& S = *C.S;
  using Idx = typename RoundWs<SM>::Idx;
  constexpr int kNone = RoundWs<SM>::kNone;
  const int N = S.X.N, T = blockDim.x, W = T / 32, nt = S.nt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slack = (RoundWs<SM>::kRoom * N - n) / (S.nrap * S.nphi), vm = (1 << S.sh) - 1;
  for (int t = tid; t < nt; t += T) C.count[t] = 0;
  __syncthreads();
#pragma unroll 1
  for (int s = tid; s < N; s += T) {
    const int t = C.W.tile(s);
    if (t != kNone) C.W.at(s) = (Idx)atomicAdd(&C.count[t], 1);
  }
  __syncthreads();
  int carry = 0;
#pragma unroll 1
  for (int base = 0; base < nt; base += T) {
    const int t = base + tid;
    const int v = t < nt && (t & vm) < S.nphi ? C.count[t] + slack : 0;
    int incl = v;
#pragma unroll 1
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += x;
    }
    if (lane == 31) S.scan_tmp[warp] = incl;
    __syncthreads();
    int pre = 0, total = 0;
#pragma unroll 1
    for (int k = 0; k < W; ++k) {
      if (k < warp) pre += S.scan_tmp[k];
      total += S.scan_tmp[k];
    }
    if (t < nt) C.start[t] = (Idx)(carry + pre + incl - v);
    carry += total;
    __syncthreads();
  }
  if (tid == 0) C.start[nt] = (Idx)carry;
  __syncthreads();
#pragma unroll 1
  for (int s = tid; s < N; s += T) {
    const int t = C.W.tile(s);
    if (t != kNone) C.W.place(C.start[t] + C.W.at(s), s, C.W.xy(s));
  }
  __syncthreads();
}

// Lane's dead node idx, taken by a step of time part m_hi (rounded up) and label
// l, into its tile's groups (lanes with the same tile go one after another).
// Groups are kept by descending M, so that a walk for times from some M on ends
// at the first that is before it.  What a jet absorbs one after another has the
// same (M, l) while its steps are chained: one group, which the jet's own
// checks pass at once.  (One list of single nodes: 25 to 90 kcycles a round on
// dense anti-kt events, most of it a jet walking over its own constituents.)
template <bool SM>
__device__ __noinline__ void round_bury(bool have, int tile, int idx, float4 g, float m_hi, int l) {
  const RoundCtx<SM> C = round_ctx<SM>();
  const int most = 2 * C.S->X.N;
  bool todo = have;
  while (__any_sync(kFull, todo)) {
    const unsigned same = __match_any_sync(kFull, todo ? tile : -1 - (int)(threadIdx.x & 31));
    if (todo && (threadIdx.x & 31) == (unsigned)(__ffs(same) - 1)) {
      todo = false;
      C.W.dgeo(idx) = g;
      int prev = -1, x = C.head[tile];
      float xm = C.head_m[tile];
#pragma unroll 1
      for (int guard = 0; x >= 0 && xm > m_hi && guard < most; ++guard) {
        const int4 r = C.W.dgrp(x);
        prev = x;
        x = r.x;
        xm = __int_as_float(r.y);
      }
      int q = x;
      float qm = xm;
      bool found = false;
#pragma unroll 1
      for (int guard = 0; q >= 0 && qm == m_hi && !found && guard < most; ++guard) {
        const int4 r = C.W.dgrp(q);
        if (r.w == l) {
          C.W.dnext(idx) = r.z;
          C.W.dgrp(q).z = idx;
          found = true;
        }
        q = r.x;
        qm = __int_as_float(r.y);
      }
      if (!found) {
        C.W.dnext(idx) = -1;
        C.W.dgrp(idx) = make_int4(x, __float_as_int(xm), idx, l);
        if (prev < 0) {
          C.head[tile] = idx;
          C.head_m[tile] = m_hi;
        } else {
          *reinterpret_cast<int2*>(&C.W.dgrp(prev)) = make_int2(idx, __float_as_int(m_hi));
        }
      }
    }
    __syncwarp();
  }
}

// D2 over one tile's groups for the new jet a of the step at time (M, l, depth)
// (see the header), from its first group x on.  The dead of a's own line (label
// l) went before it.
template <bool SM>
__device__ __noinline__ bool round_d2(int x, int a, double M, int l, int depth) {
  const RoundCtx<SM> C = round_ctx<SM>();
  const EventCtx& X = C.S->X;
  const float m_lo = __double2float_rd(M), wa = round_wlo(C.W.wlo(a)), r2hi = C.S->r2hi, ilo = X.ilo;
  const float2 ga = C.W.xy(a);
  const Bound bd = X.bd;
  bool bad = false;
#pragma unroll 1
  for (int guard = 0; x >= 0 && guard < 2 * X.N; ++guard) {
    const int4 r = C.W.dgrp(x);
    if (r.w != l) {
      int y = r.z;
#pragma unroll 1
      for (int g2 = 0; y >= 0 && g2 < 2 * X.N; ++g2) {
        const float4 dg = C.W.dgeo(y);
        float lo, hi;
        dr2_32(dg.x, dg.y, ga.x, ga.y, bd, lo, hi);
        const float plo = __fmul_rd(__fmul_rd(__fmul_rd(fminf(wa, dg.z), lo), ilo), 0.99999976158142089844f);
        if (lo <= r2hi && !(plo > dg.w)) {
          const RoundRec q = C.W.rec(y >> 1);
          if (time_less(RoundTime{M, l, depth}, RoundTime{q.M, q.l, q.depth})) {
            bad = true;
            // (both positive: ordered as integers)
            atomicMin(&C.S->early, (unsigned long long)q.round << 32 | (unsigned)(y >> 1));
            atomicMax(&C.S->hold, __float_as_int(m_lo));
          }
        }
        y = C.W.dnext(y);
      }
    }
    if (__int_as_float(r.y) < m_lo) break;
    x = r.x;
  }
  return bad;
}

// What came too early (whole CTA): the first such step and all of its line (the
// steps of the same M and l, which a jet takes one after another: while its first
// one stands, the others' turn seems to have come).  Their first round is where to
// go back to, and their slots are held.  (Back to that one step, with its slot
// held: up to ten conflicts with one line, each a few of its steps further back.)
template <bool SM>
__device__ __noinline__ void round_line() {
  const RoundCtx<SM> C = round_ctx<SM>();
  RoundShared& S = *C.S;
  if (S.early == ~0ull) return;
  const RoundRec first = C.W.rec((int)(unsigned)S.early);
#pragma unroll 1
  for (int s = threadIdx.x; s < S.X.N; s += blockDim.x) {
    if (C.W.tile(s) != (typename RoundWs<SM>::Idx)RoundWs<SM>::kNone) continue;
    const RoundRec r = C.W.rec(s);
    if (r.M != first.M || r.l != first.l) continue;
    atomicMin(&S.back, r.round);
    atomicMax(reinterpret_cast<int*>(&C.W.slots[s].hold), S.hold);
    if (r.a >= 0) atomicMax(reinterpret_cast<int*>(&C.W.slots[r.a].hold), S.hold);
  }
  __syncthreads();
}

// What the time of a step is made of: of c and of its partner j.
struct RoundPair {
  double wc, wj, mc, mj;
  double2 pc, pj;
  int2 lc, lj;
  int fj;
};

template <bool SM>
__device__ __forceinline__ RoundPair round_pair(const RoundWs<SM>& W, int c, int j) {
  return RoundPair{W.w(c), W.w(j), W.tm(c), W.tm(j), W.pos(c), W.pos(j), W.tl(c), W.tl(j), (int)W.nn(j)};
}

// The step of slot c with partner j (-1: none): its key, its time and whether it
// follows that of c or of j.
struct RoundStep {
  int c, j;
  double key;
  RoundTime t;
  bool chained, from_j;
};

template <bool SM>
__device__ __forceinline__ RoundStep round_step(int c, int j, const RoundPair& p, double inv_r2) {
  const bool mutual = j >= 0 && (p.fj & RoundWs<SM>::kPair) && (p.fj & RoundWs<SM>::kSlotMask) == c;
  RoundStep s{c, j, p.wc, {}, false, false};
  RoundTime tc{p.mc, p.lc.x, p.lc.y}, tj{-2.0, -1, 0};
  if (j >= 0) {
    s.key = pair_distance(p.wc, p.wj, dr2_64(p.pc.x, p.pc.y, p.pj.x, p.pj.y), inv_r2);
    tj = RoundTime{p.mj, p.lj.x, p.lj.y};
    if (p.wj <= s.key && p.wj < p.wc) {
      // a partner at R, up to FP32: its promotion goes first
      s.c = j;
      s.j = -1;
      s.key = p.wj;
      tc = tj;
      tj = RoundTime{-2.0, -1, 0};
    }
  }
  s.from_j = time_less(tc, tj);
  const RoundTime tp = s.from_j ? tj : tc;
  s.t = RoundTime{s.key, mutual && s.j >= 0 ? min(c, j) : s.c, 0};
  s.chained = s.t.M < tp.M || (s.t.M == tp.M && s.t.l <= tp.l);
  if (s.chained) s.t = RoundTime{tp.M, tp.l, tp.depth + 1};
  return s;
}

// Whether the step of slots c and j, of time P, has to wait: they are held until
// nothing with a time up to `hold` (0: not held) is left; the earliest step of all
// never is.  The bounds on times are good to 2^-15.  (Asked only after a conflict.)
template <bool SM>
__device__ __noinline__ bool round_held(int c, int j, float P) {
  const RoundCtx<SM> C = round_ctx<SM>();
  const float hold = fmaxf(C.W.slots[c].hold, C.W.slots[j].hold), p_min = __uint_as_float(C.S->p_min);
  return hold > 0.0f && P >= hold * (1.0f - 0x1p-13f) && p_min < P && p_min <= hold * (1.0f + 0x1p-13f);
}

// The order of steps: those of the same time follow the same one, the smallest
// key first.
__device__ __forceinline__ bool round_earlier(const RoundTime& x, double kx, int cx, const RoundTime& y, double ky,
                                              int cy) {
  if (time_less(x, y)) return true;
  if (time_less(y, x)) return false;
  return kx < ky || (kx == ky && cx < cy);
}

// A slot with the earliest step of all, per warp, into S.targets (whole CTA); P
// is within 2^-15 of the time's M.
template <bool SM>
__device__ __noinline__ void round_pick() {
  const RoundCtx<SM> C = round_ctx<SM>();
  RoundShared& S = *C.S;
  using Ws_ = RoundWs<SM>;
  const float lim = __uint_as_float(S.p_min) * (1.0f + 0x1p-13f);
  RoundStep best{};
  int slot = -1;
#pragma unroll 1
  for (int s = threadIdx.x; s < S.X.N; s += blockDim.x) {
    if (C.W.tile(s) == (typename Ws_::Idx)Ws_::kNone || !(C.W.key(s).y <= lim)) continue;
    const int f = C.W.nn(s), j = f & Ws_::kPair ? f & Ws_::kSlotMask : -1;
    const RoundStep q = round_step<SM>(s, j, round_pair(C.W, s, j >= 0 ? j : s), S.X.inv_r2);
    if (slot < 0 || round_earlier(q.t, q.key, s, best.t, best.key, slot)) {
      best = q;
      slot = s;
    }
  }
#pragma unroll 1
  for (int o = 16; o; o >>= 1) {
    RoundTime t;
    t.M = __shfl_xor_sync(kFull, best.t.M, o);
    t.l = __shfl_xor_sync(kFull, best.t.l, o);
    t.depth = __shfl_xor_sync(kFull, best.t.depth, o);
    const double key = __shfl_xor_sync(kFull, best.key, o);
    const int other = __shfl_xor_sync(kFull, slot, o);
    if (other >= 0 && (slot < 0 || round_earlier(t, key, other, best.t, best.key, slot))) {
      best.t = t;
      best.key = key;
      slot = other;
    }
  }
  if ((threadIdx.x & 31) == 0 && slot >= 0) round_target(S, slot);
}

// Of the round's steps only the earliest stays (one thread).
template <bool SM>
__device__ __noinline__ void round_earliest() {
  const RoundCtx<SM> C = round_ctx<SM>();
  RoundShared& S = *C.S;
  int b = 0;
#pragma unroll 1
  for (int i = 1; i < min(S.n_fire, kRoundSteps); ++i)
    if (round_earlier(RoundTime{S.M[i], S.l[i], S.depth[i]}, S.key[i], S.c[i],
                      RoundTime{S.M[b], S.l[b], S.depth[b]}, S.key[b], S.c[b]))
      b = i;
  if (S.new_u[b]) S.conflict[0] = 1;
  S.c[0] = S.c[b];
  S.j[0] = S.j[b];
  S.key[0] = S.key[b];
  S.M[0] = S.M[b];
  S.l[0] = S.l[b];
  S.depth[0] = S.depth[b];
  S.thr_c[0] = S.thr_c[b];
  S.thr_j[0] = S.thr_j[b];
  S.tile_c[0] = S.tile_c[b];
  S.tile_j[0] = S.tile_j[b];
  S.xy_c[0] = S.xy_c[b];
  S.xy_j[0] = S.xy_j[b];
  S.wlo[0] = S.wlo[b];
  S.n_fire = min(S.n_fire, 1);
  S.n_targets = 0;
}

// Takes back the steps of rounds r0 and later (whole CTA): the slots they removed
// return, those they merged into get back what the first such step saved, and the
// groups of the dead are made again from the others' (a warp per 1 / W of the
// tiles).  Lists, neighbours and minima are to be made again.  Leaves the number
// of live slots in S.alive.
template <bool SM>
__device__ __noinline__ void round_undo(int r0) {
  const RoundCtx<SM> C = round_ctx<SM>();
  RoundShared& S = *C.S;
  using Idx = typename RoundWs<SM>::Idx;
  constexpr int kNone = RoundWs<SM>::kNone;
  const int N = S.X.N, T = blockDim.x, W = T / 32, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto undone = [&](int s) { return C.W.tile(s) == kNone && C.W.rec(s).round >= r0 && C.W.rec(s).a >= 0; };
  for (int s = tid; s < N; s += T) C.W.slots[s].parent = 0x7fffffff;
  for (int t = tid; t < S.nt; t += T) {
    C.head[t] = -1;
    C.head_m[t] = 0.0f;
  }
  if (tid == 0) S.alive = 0;
  __syncthreads();
#pragma unroll 1
  for (int s = tid; s < N; s += T)
    if (undone(s)) atomicMin(&C.W.slots[C.W.rec(s).a].parent, C.W.rec(s).round);
  __syncthreads();
#pragma unroll 1
  for (int s = tid; s < N; s += T) {
    if (!undone(s)) continue;
    const int a = C.W.rec(s).a;
    if (C.W.slots[a].parent != C.W.rec(s).round) continue;
    const RoundDead& D = C.W.dead[s];
    for (int q = 0; q < 4; ++q) C.W.p4(q, a) = D.p[q];
    C.W.w(a) = D.w;
    C.W.pos(a) = D.pos;
    C.W.tm(a) = D.tm;
    C.W.tl(a) = D.tl;
    C.W.tlo(a) = fmaxf(__double2float_rd(D.tm), 0.0f);
    C.W.xy(a) = make_float2(__double2float_rn(D.pos.x), __double2float_rn(D.pos.y));
    C.W.wlo(a) = round_weight(D.w);
  }
  __syncthreads();
  int alive = 0;
#pragma unroll 1
  for (int s = tid; s < N; s += T) {
    if (C.W.tile(s) == kNone && C.W.rec(s).round < r0) continue;
    const double2 p = C.W.pos(s);
    C.W.tile(s) = (Idx)((round_u(S, p.x) << S.sh) + round_v(S, p.y));
    ++alive;
  }
  alive = __reduce_add_sync(kFull, alive);
  if (lane == 0) atomicAdd(&S.alive, alive);
  __syncthreads();
#pragma unroll 1
  for (int s0 = 0; s0 < N; s0 += 32) {
    const int s = s0 + lane;
    const bool dead = s < N && C.W.tile(s) == kNone;
    const RoundRec r = C.W.rec(dead ? s : s0);
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
      const float4 g = C.W.dgeo(2 * (dead ? s : s0) + q);
      const int t = dead && (!q || r.a >= 0) ? (round_u(S, g.x) << S.sh) + round_v(S, g.y) : -1;
      const bool mine = t >= 0 && t % W == warp;
      if (__any_sync(kFull, mine)) round_bury<SM>(mine, mine ? t : 0, 2 * s + q, g, __double2float_ru(r.M), r.l);
    }
  }
  if (tid == 0) {
    S.conflict[0] = S.conflict[1] = S.conflict[2] = 0;
    S.n_cand = S.n_fire = S.n_targets = S.overflow = 0;
    S.p_min = kRoundNone;
    S.task[0] = S.task[1] = 0;
  }
  __syncthreads();
}

// Initial neighbours: a thread per slot, or (dense) a warp per tile -- a lane per
// member, the window's slots gathered by the lanes and passed around.
template <bool SM>
__device__ __forceinline__ void round_init(const RoundCtx<SM>& C, bool dense) {
  const RoundShared& S = *C.S;
  const int lane = threadIdx.x & 31, N = S.X.N;
  const Bound bd = S.X.bd;
  if (!SM && dense) {
#pragma unroll 1
    for (int tile = threadIdx.x >> 5; tile < S.nt; tile += blockDim.x >> 5) {
      const int st0 = C.start[tile], m0 = C.count[tile];
      if (!m0) continue;
      const RoundBox b = round_box(S, tile, tile);
      const int nb = b.nu * b.nv;
#pragma unroll 1
      for (int i0 = 0; i0 < m0; i0 += 32) {
        const bool have = i0 + lane < m0;
        const int t = C.W.members[st0 + (have ? i0 + lane : i0)];
        const float2 gt = C.W.xy(t);
        Cert c = cert_empty();
        // its own tile, then those that can hold something closer for a lane
#pragma unroll 1
        for (int k = -1; k < nb; ++k) {
          const int tt = k < 0 ? tile : box_tile(S, b, k);
          if (k >= 0) {
            const float d = tile_d2(S, gt, tt >> S.sh, tt & ((1 << S.sh) - 1)) * 0.999f - 1e-6f;
            if (tt == tile || !__any_sync(kFull, have && d <= c.u1)) continue;
          }
          const int st = C.start[tt], m = C.count[tt];
#pragma unroll 1
          for (int q0 = 0; q0 < m; q0 += 32) {
            const int left = min(m - q0, 32);
            const int iq = st + q0 + (lane < left ? lane : 0);
            const int uq = C.W.members[iq];
            const float2 gq = C.W.entry(uq, iq);
#pragma unroll 4
            for (int q = 0; q < left; ++q) {
              const int u = __shfl_sync(kFull, uq, q);
              float lo, hi;
              dr2_32(gt.x, gt.y, __shfl_sync(kFull, gq.x, q), __shfl_sync(kFull, gq.y, q), bd, lo, hi);
              if (u != t) cert_add(c, lo, hi, u);
            }
          }
        }
        round_settle<SM>(have, true, t, c, 0);
      }
    }
    return;
  }
#pragma unroll 1
  for (int s0 = threadIdx.x & ~31; s0 < N; s0 += blockDim.x) {
    const int t = s0 + lane;
    const int tile = t < N ? C.W.tile(t) : (typename RoundWs<SM>::Idx)RoundWs<SM>::kNone;
    const bool have = t < N && tile != RoundWs<SM>::kNone;
    Cert c = cert_empty();
    if (have) {
      const RoundBox b = round_box(S, tile, tile);
      const int nb = b.nu * b.nv;
      const float2 gt = C.W.xy(t);
#pragma unroll 1
      for (int k = 0; k < nb; ++k) {
        const int tt = box_tile(S, b, k);
        const int st = C.start[tt], m = C.count[tt];
#pragma unroll 2
        for (int i = 0; i < m; ++i) {
          const int u = C.W.members[st + i];
          const float2 gu = C.W.entry(u, st + i);
          float lo, hi;
          dr2_32(gt.x, gt.y, gu.x, gu.y, bd, lo, hi);
          if (u != t) cert_add(c, lo, hi, u);
        }
      }
    }
    __syncwarp();
    round_settle<SM>(have, true, t, c, 0);
  }
}

__device__ __forceinline__ float plain_dr2(float2 a, float2 b) {
  const float dr = a.x - b.x;
  float dp = fabsf(a.y - b.y);
  dp = fminf(dp, kTwoPiF - dp);
  return dr * dr + dp * dp;
}

// Phase B for the steps, by groups of G lanes: D1, and the slots whose neighbour
// is taken.  With few steps their windows are cut in parts.
template <bool SM>
__device__ __forceinline__ void round_phase_b(const RoundCtx<SM>& C, int F, int G, int parts) {
  using Ws_ = RoundWs<SM>;
  RoundShared& S = *C.S;
  const Ws_& Wk = C.W;
  const int lane = threadIdx.x & 31;
  const Bound bd = S.X.bd;
  const float ilo = S.X.ilo, r2hi = S.r2hi, far2 = S.far2;
#pragma unroll 1
  for (;;) {
    int i = 0;
    if (lane == 0) i = atomicAdd(&S.task[0], 32 / G);
    i = __shfl_sync(kFull, i, 0);
    if (i >= F * parts) break;
    const int part = i % parts;  // (several parts: G = 32)
    i = G == 32 ? i / parts : i + lane / 8;
    const bool have = i < F;
    const int at = have ? i : 0, c = S.c[at], j = have ? S.j[at] : -1;
    const float2 gc = S.xy_c[at], gj = S.xy_j[at];
    const float wc = S.wlo[at].x, wj = S.wlo[at].y;
    RoundBox b{0, 0, 0, 1};
    double M = 0.0, thr_c = 0.0, thr_j = 0.0;
    if (have) {
      M = S.M[i];
      thr_c = S.thr_c[i];
      thr_j = S.thr_j[i];
      b = round_box(S, S.tile_c[i], S.tile_j[i]);
    }
    const float tc_hi = __double2float_ru(thr_c), tj_hi = __double2float_ru(thr_j);
    struct Slot {
      float2 g;
      float w;
      int nn;
    };
    bool bad = false;
    const int nb = b.nu * b.nv;
    for_tiles(C, b, nb * part / parts, nb * (part + 1) / parts, G, gc, gj,
            [&](int y, float2 g) { return Slot{g, Wk.wlo(y), Wk.nn(y)}; },
            [&](int y, const Slot& s) {
              if (y == c || y == j) return;
              const int nn = s.nn & Ws_::kSlotMask;
              if (nn == c || (j >= 0 && nn == j)) {
                Wk.nn(y) = (typename Ws_::Idx)(s.nn | Ws_::kTarget);
                round_target(S, y);
              }
              // beyond R of c and of j (round_far2)?
              if (fminf(plain_dr2(gc, s.g), plain_dr2(gj, s.g)) > far2) return;
              const float w = round_wlo(s.w);
#pragma unroll 1
              for (int q = 0; q < 2; ++q) {
                const float2 gx = q ? gj : gc;
                float lo, hi;
                dr2_32(gx.x, gx.y, s.g.x, s.g.y, bd, lo, hi);
                const float plo =
                    __fmul_rd(__fmul_rd(__fmul_rd(fminf(q ? wj : wc, w), lo), ilo), 0.99999976158142089844f);
                if (!(lo > r2hi) && !(plo > (q ? tj_hi : tc_hi)))
                  bad |= round_d1_exact<SM>(q ? j : c, y, q ? thr_j : thr_c, M);
                if (j < 0) break;
              }
            });
    if (bad) S.conflict[1] = 1;
  }
}

// Phase D for one step that made jet a (groups of G lanes): the jet's window.
template <bool SM>
__device__ __forceinline__ void round_new_jet(const RoundCtx<SM>& C, bool have, int i, int G,
                                              int part, int parts) {
  using Ws_ = RoundWs<SM>;
  RoundShared& S = *C.S;
  const Ws_& Wk = C.W;
  const int lane = threadIdx.x & 31;
  const Bound bd = S.X.bd;
  const int a = have ? min(S.c[i], S.j[i]) : 0;
  const int tile = have ? (S.new_u[i] << S.sh) + S.new_v[i] : 0;
  RoundBox b = round_box(S, tile, tile);
  if (!have) b.nu = 0;
  const float2 ga = make_float2(__double2float_rn(S.rap[have ? i : 0]), __double2float_rn(S.phi[have ? i : 0]));
  struct Slot {
    float2 g;
    float nhi;
    int nn;
  };
  Cert ca = cert_empty();
  const int nb = b.nu * b.nv;
  for_tiles(C, b, nb * part / parts, nb * (part + 1) / parts, G, ga, ga,
          [&](int y, float2 g) { return Slot{g, Wk.nhi(y), Wk.nn(y)}; },
          [&](int y, const Slot& s) {
            if (y == a) return;
            float lo, hi;
            dr2_32(s.g.x, s.g.y, ga.x, ga.y, bd, lo, hi);
            cert_add(ca, lo, hi, y);
            // not closer, or searched anyway?
            if (!(lo > s.nhi) && !(s.nn & Ws_::kTarget)) round_offer<SM>(y, a, lo, hi, s.nhi);
          });
  ca = cert_group(ca, G);
  if (parts > 1 && !round_join(C, ca, i, part, parts)) return;
  round_settle<SM>(have, (lane & (G - 1)) == 0, a, ca, Ws_::kTarget);
}

// Records of an event with its slots in shared memory in time order: bitonic sort
// there (in the room of the tile arrays and of the slots' state up to `members`,
// which takes the order: 30 bytes a slot and more, for 14 a record; the slots are a
// power of two).  Labels and depths are below 4096.  4000 particles: 0.2 M cycles,
// 0.55 M in the workspace.
__device__ __forceinline__ void round_sort_smem(const RoundCtx<true>& C, int N, int n2,
                                                RoundWs<true>::Idx* order) {
  static_assert(kRoundSlotBytes - RoundWs<true>::kRoom * sizeof(RoundWs<true>::Idx) >= 14, "room for the sort");
  const int T = blockDim.x;
  unsigned long long* M = reinterpret_cast<unsigned long long*>(C.tmin);
  unsigned* sec = reinterpret_cast<unsigned*>(M + n2);
  unsigned short* id = reinterpret_cast<unsigned short*>(sec + n2);
#pragma unroll 1
  for (int s = threadIdx.x; s < n2; s += T) {
    M[s] = ~0ull;
    sec[s] = kRoundNone;
    id[s] = (unsigned short)s;
    if (s < N) {
      const RoundRec r = C.W.rec(s);
      M[s] = dbits(r.M);  // non-negative: ordered as integers
      sec[s] = ((unsigned)r.l << 12) | (unsigned)r.depth;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int size = 2; size <= n2; size <<= 1) {
#pragma unroll 1
    for (int stride = size >> 1, sh = 31 - __clz(size >> 1); stride > 0; stride >>= 1, --sh) {
#pragma unroll 2
      for (int k = threadIdx.x; k < n2 / 2; k += T) {
        const int i = ((k >> sh) << (sh + 1)) + (k & (stride - 1)), j = i + stride;
        const bool up = (i & size) == 0;
        const unsigned long long x = M[i], y = M[j];
        const unsigned sx = sec[i], sy = sec[j];
        const bool gt = x > y || (x == y && sx > sy);
        if (gt == up) {
          M[i] = y;
          M[j] = x;
          sec[i] = sy;
          sec[j] = sx;
          const unsigned short t = id[i];
          id[i] = id[j];
          id[j] = t;
        }
      }
      __syncthreads();
    }
  }
  for (int s = threadIdx.x; s < N; s += T) order[s] = id[s];
  __syncthreads();
}

// Any number of records, in the workspace.  The first stride of a size pairs
// mirrored entries, so that every run ascends and the missing entries past N
// act as the largest.
__device__ __forceinline__ void round_sort(const RoundCtx<false>& C, int N, int n2, RoundWs<false>::Idx* order) {
  using Idx = RoundWs<false>::Idx;
  const int T = blockDim.x;
  for (int s = threadIdx.x; s < N; s += T) order[s] = (Idx)s;
  __syncthreads();
#pragma unroll 1
  for (int size = 2; size <= n2; size <<= 1) {
#pragma unroll 1
    for (int stride = size >> 1, sh = 31 - __clz(size >> 1); stride > 0; stride >>= 1, --sh) {
      const bool flip = stride == size >> 1;
#pragma unroll 2
      for (int k = threadIdx.x; k < n2 / 2; k += T) {
        const int base = (k >> sh) << (sh + 1), r = k & (stride - 1);
        const int lo = base + r, hi = flip ? base + 2 * stride - 1 - r : lo + stride;
        if (hi < N) {
          const Idx x = order[lo], y = order[hi];
          const RoundRec& rx = C.W.rec(x);
          const RoundRec& ry = C.W.rec(y);
          if (time_less(RoundTime{ry.M, ry.l, ry.depth}, RoundTime{rx.M, rx.l, rx.depth})) {
            order[lo] = y;
            order[hi] = x;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Clusters event e; false: a conflict (nothing of the event's outputs was
// written).  S.tiles, cells and slots are set.
template <int T, bool SM>
__device__ __forceinline__ bool cluster_event_rounds(RoundShared& S, const BatchArgs& A, int e) {
  constexpr int W = T / 32;
  using Ws_ = RoundWs<SM>;
  using Idx = typename Ws_::Idx;
  constexpr int kNone = Ws_::kNone;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float inf = __int_as_float(0x7f800000);
  FJG_PH(long long ph[kPhSlots - kPhRSetup] = {}; long long ph_t = clock64();
         auto mark = [&](int slot) { const long long now = clock64(); ph[slot - kPhRSetup] += now - ph_t; ph_t = now; };)
  int64_t off;
  int N;
  event_range(A, e, off, N);
  const int algo = A.algo ? A.algo[e] : A.algo_all;
  const double R = A.radius ? A.radius[e] : A.r_all;
  if (tid == 0) {
    S.X.N = N;
    S.X.algo = algo;
    S.X.inv_r2 = 1.0 / (R * R);
    S.X.ilo = __double2float_rd(S.X.inv_r2);
    S.X.ihi = __double2float_ru(S.X.inv_r2);
    S.ws = A.round_ws + off * kRoundBytesPerParticle;
    S.r2hi = __double2float_ru(R * R) * 1.0001f;
  }
  __syncthreads();
  const RoundCtx<SM> C = round_ctx<SM>();
  const Ws_& Wk = C.W;

  // ---- load and kinematics
  double rlo = 1e300, rhi = -1e300, amax = 0.0;
  bool refused = false;  // left to the other kernels (round_refuses)
#pragma unroll 1
  for (int s = tid; s < N; s += T) {
    const double* p = A.p4 + (off + s) * A.p4_stride;
    const double px = p[0], py = p[1], pz = p[2], E = p[3];
    const Kin kin = kinematics(px, py, pz, E, algo);
    Wk.p4(0, s) = px;
    Wk.p4(1, s) = py;
    Wk.p4(2, s) = pz;
    Wk.p4(3, s) = E;
    Wk.w(s) = kin.w;
    Wk.pos(s) = make_double2(kin.rap, kin.phi);
    Wk.xy(s) = make_float2(__double2float_rn(kin.rap), __double2float_rn(kin.phi));
    Wk.wlo(s) = round_weight(kin.w);
    Wk.tlo(s) = 0.0f;
    Wk.tm(s) = -1.0;
    Wk.slots[s].hold = 0.0f;
    Wk.tl(s) = make_int2(-1, 0);
    rlo = fmin(rlo, kin.rap);
    rhi = fmax(rhi, kin.rap);
    amax = fmax(amax, fabs(kin.rap));
    refused |= round_refuses(kin.w) || round_refuses_rap(kin.rap);
  }
#pragma unroll 1
  for (int o = 16; o; o >>= 1) {
    rlo = fmin(rlo, __shfl_xor_sync(kFull, rlo, o));
    rhi = fmax(rhi, __shfl_xor_sync(kFull, rhi, o));
    amax = fmax(amax, __shfl_xor_sync(kFull, amax, o));
  }
  if (lane == 0) {
    S.red[0][warp] = rlo;
    S.red[1][warp] = rhi;
    S.red[2][warp] = amax;
  }
  for (int k = tid; k < kRoundMaxTiles / 32; k += T) S.dirty_bits[k] = 0;
  for (int k = tid; k < kRoundSmemMaxN / 32; k += T) S.taken[k] = S.claimed[k] = 0;
  if (tid < 16) S.lut[tid] = tid ? (65536 + tid - 1) / tid : 0;
  if (__syncthreads_or(refused)) {
    FJG_PH(if (A.phase && tid == 0) atomicAdd(A.phase + kPhRRetries, 1ull);)
    return false;
  }
  if (tid == 0) {
    double lo = 1e300, hi = -1e300, rmax = 0.0;
#pragma unroll 1
    for (int k = 0; k < W; ++k) {
      lo = fmin(lo, S.red[0][k]);
      hi = fmax(hi, S.red[1][k]);
      rmax = fmax(rmax, S.red[2][k]);
    }
    S.X.bd = make_bound(rmax);
    S.far2 = round_far2(S.r2hi, rmax);
    lo = fmax(lo, -15.0);
    hi = fmin(hi, 15.0);
    if (!(hi >= lo)) hi = lo;
    // side: at least R / 2, so that the 5x5 window holds R; coarser where that
    // would give more tiles than there is room for, or than 1.5 per particle
    // (empty tiles only cost)
    int cap = N + N / 2;
    cap = cap > S.tiles ? S.tiles : cap;
    cap = cap < 1 ? 1 : cap;
    const double side_min = 0.5 * R * (1.0 + 1e-4) + 1e-5;
    const double area = fmax(hi - lo, side_min) * 6.283185307179586;
    const double side = fmax(side_min, sqrt(area / (double)cap));
    int nphi = (int)fmin(floor(6.283185307179586 / side), 4096.0);
    nphi = nphi < 1 ? 1 : nphi;
    int nrap = (int)fmin(floor((hi - lo) / side), 4096.0);
    nrap = nrap < 1 ? 1 : nrap;
    int sh = 0;
#pragma unroll 1
    for (;;) {  // ends: one tile always has room
      sh = 0;
      while ((1 << sh) < nphi) ++sh;
      if ((nrap << sh) <= S.tiles && nrap * nphi <= cap &&
          (nrap + 2 * kRoundFrame) * (nphi + 2 * kRoundFrame) <= S.cells)
        break;
      if (nrap >= nphi)
        nrap = nrap > 8 ? nrap - nrap / 8 : nrap - 1;
      else
        nphi = nphi > 8 ? nphi - nphi / 8 : nphi - 1;
    }
    S.nrap = nrap;
    S.nphi = nphi;
    S.sh = sh;
    S.nt = nrap << sh;
    S.pw = nphi + 2 * kRoundFrame;
    S.rmin = lo;
    S.inv_side_r = (double)nrap / fmax(hi - lo, side);
    S.inv_side_phi = (double)nphi / 6.283185307179586;
    S.rmin32 = (float)lo;
    S.side_r = (float)(1.0 / S.inv_side_r);
    S.side_phi = (float)(1.0 / S.inv_side_phi);
    S.conflict[0] = S.conflict[1] = S.conflict[2] = 0;
    S.overflow = S.hopeless = S.backs = S.ties = S.care = S.care_until = 0;
    S.p_min = kRoundNone;
    S.reach = algo != -1 ? kRoundReachKt : N > kRoundLargeFrom ? kRoundReachLarge : kRoundReach;
    S.n_cand = S.n_fire = S.n_targets = S.n_dirty = 0;
    S.task[0] = S.task[1] = 0;
  }
  __syncthreads();
  FJG_PH(mark(kPhRKin);)
  const int nt = S.nt, pw = S.pw, sh = S.sh, nphi = S.nphi;
  for (int t = tid; t < nt; t += T) {
    C.head[t] = -1;
    C.head_m[t] = 0.0f;
  }
  for (int t = tid; t < (S.nrap + 2 * kRoundFrame) * pw; t += T) C.tmin[t] = C.row[t] = kRoundNone;
#pragma unroll 1
  for (int s = tid; s < N; s += T) {
    const double2 p = Wk.pos(s);
    Wk.tile(s) = (Idx)((round_u(S, p.x) << sh) + round_v(S, p.y));
  }
  __syncthreads();

  int n = N, round = 0;
#pragma unroll 1
  for (;;) {
  round_lists<SM>(n);
  // ---- neighbours (round_set marks tiles as changed: cleared after)
  round_init(C, n >= kRoundDense * nt);
  __syncthreads();
  if (round == 0 && S.ties > 1 + N / kRoundTies) {
    FJG_PH(if (A.phase && tid == 0) atomicAdd(A.phase + kPhRRetries, 1ull);)
    return false;
  }
  for (int t = tid; t < nt; t += T) round_summary_thread<SM>(t);
  for (int k = tid; k < kRoundMaxTiles / 32; k += T) S.dirty_bits[k] = 0;
  __syncthreads();
  if (tid == 0) {
    S.n_dirty = 0;
    S.back = 0x7fffffff;
    S.early = ~0ull;
    S.hold = 0;
  }
  FJG_PH(mark(kPhRSetup);)

  // ---- rounds
  const float side_r = S.side_r, side_phi = S.side_phi;
  const float rmin = S.rmin32, inv_side = 1.0f / fminf(side_r, side_phi);
#pragma unroll 1
  for (; n > 0; ++round) {
    const bool dense = !SM && n >= kRoundDense * nt;
    const int care = round < S.care_until ? S.care : 0;
    // A: candidates.  Smallest P of five tiles along the row, then of five
    // rows (empty tiles hold the largest value)
#pragma unroll (SM ? 1 : 4)
    for (int t = tid; t < nt; t += T) {
      const int u = t >> sh, v = t & ((1 << sh) - 1);
      if (v >= nphi) continue;
      const int k = (u + kRoundFrame) * pw + kRoundFrame + v;
      C.row[k] = min(min(min(C.tmin[k - 2], C.tmin[k - 1]), min(C.tmin[k + 1], C.tmin[k + 2])), C.tmin[k]);
    }
    if (!SM)
      for (int k = tid; k < (S.nrap + 2 * kRoundFrame) * pw; k += T) C.near[k] = C.tmin[k];
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < nt; t += T) {
      const int u = t >> sh, v = t & ((1 << sh) - 1);
      if (v >= nphi) continue;
      const int k = (u + kRoundFrame) * pw + kRoundFrame + v;
      const unsigned me = C.tmin[k];
      if (me == kRoundNone) continue;
      if (S.backs) atomicMin(&S.p_min, me);
      if (!SM) {
        // a step also counts where its partner is: a hard jet's own key may
        // belong to a later step (its neighbour is younger) while an earlier
        // one takes it from the far side of its reach
        const int tj = C.beside[t];
        if (tj != t) {
          const int vj = tj & ((1 << sh) - 1);
          unsigned* cell = C.near + ((tj >> sh) + kRoundFrame) * pw + kRoundFrame;
          atomicMin(cell + vj, me);
          // (copies across the azimuth seam: at most one each way in the frame of ten tiles or more)
          if (vj >= nphi - kRoundFrame && vj - nphi >= -kRoundFrame) atomicMin(cell + vj - nphi, me);
          if (vj < kRoundFrame) atomicMin(cell + vj + nphi, me);
        }
      }
      if (me == min(min(min(C.row[k - 2 * pw], C.row[k - pw]), min(C.row[k + pw], C.row[k + 2 * pw])), C.row[k])) {
        const int q = atomicAdd(&S.n_cand, 1);
        if (q < kRoundMaxCand) S.cand[q] = (unsigned short)t;
      }
    }
    if (!SM && tid < kRoundSplit) S.parts_done[tid] = 0;
    for (int k = tid; k < (SM ? (N + 31) / 32 : kRoundSmemMaxN / 32); k += T) S.taken[k] = S.claimed[k] = 0;
    __syncthreads();
    FJG_PH(mark(kPhRCand);)
    if (care == 2) {
      round_pick<SM>();
      __syncthreads();
    }
    const int nc = care == 2 ? min(S.n_targets, kRoundSteps) : min(S.n_cand, kRoundMaxCand);
    const float range = (care ? kRoundReachWide : S.reach) * (float)R;
    // range test, eight lanes per candidate, and the keys, times and thresholds
    // of the steps that pass
#pragma unroll 1
    for (int k0 = 4 * warp; k0 < nc; k0 += 4 * W) {
      const int k = k0 + lane / 8;
      const int kk = k < nc ? k : k0, t = care == 2 ? (int)Wk.tile(S.targets[kk]) : S.cand[kk];
      const int u = t >> sh, v = t & ((1 << sh) - 1);
      const int cell = (u + kRoundFrame) * pw + kRoundFrame + v;
      const unsigned me = C.tmin[cell];
      int c = care == 2 ? S.targets[kk] : (int)C.slot[t];
      const int fc = Wk.nn(c);
      int j = fc & Ws_::kPair ? fc & Ws_::kSlotMask : -1;
      const float2 gc = Wk.xy(c);
      const float ckey = Wk.key(c).x;
      // distance within which an earlier step could matter: to c, or to its
      // partner as far from c as that is
      const float beside = j >= 0 ? sqrtf(Wk.nhi(c)) : 0.0f, lim = range + beside;
      float near2 = lim * lim;
      if (algo != -1) {
        float w = round_wlo(Wk.wlo(c));
        if (j >= 0) w = fminf(w, round_wlo(Wk.wlo(j)));
        const float l = range * sqrtf(fminf(1.0f, __uint_as_float(me) / (0.7f * w))) + beside;
        near2 = l * l;
      }
      const float fu = (gc.x - rmin) - u * side_r, fv = gc.y - v * side_phi;  // within its tile
      const float lim2 = lim * lim;
      const int far = min((int)(lim * inv_side) + 1, kRoundFrame), side = 2 * far + 1, lut = S.lut[side];
      // what a step that passes needs (in the workspace: loaded meanwhile)
      const int jc = j >= 0 ? j : c;
      RoundPair pair;
      if (!SM) pair = round_pair(Wk, c, jc);
      bool blocked = false;
#pragma unroll 1
      for (int i = lane & 7; i < side * side && care != 2; i += 8) {
        const int row = (i * lut) >> 16, du = row - far, dv = i - side * row - far;
        const unsigned o = C.near[cell + du * pw + dv];
        if (o > me) continue;
        const float dr = du > 0 ? du * side_r - fu : du < 0 ? fu - (du + 1) * side_r : 0.0f;
        const float dp = dv > 0 ? dv * side_phi - fv : dv < 0 ? fv - (dv + 1) * side_phi : 0.0f;
        const float d2 = dr * dr + dp * dp;
        if (d2 > lim2) continue;
        int ov = v + dv;
        ov = ov < 0 ? ov + nphi : ov >= nphi ? ov - nphi : ov;
        if (d2 > near2) {  // (kt, C/A) near enough for the other one's weight?
          if (o == me || ov < 0 || ov >= nphi) continue;
          const int so = C.slot[((u + du) << sh) + ov];
          if (so == kNone) continue;  // (a step counted at its partner)
          const float l = range * sqrtf(fminf(1.0f, __uint_as_float(me) / (0.7f * round_wlo(Wk.wlo(so))))) + beside;
          blocked |= d2 <= l * l;
        } else if (o < me) {
          blocked = true;
        } else if (SM || o == C.tmin[cell + du * pw + dv]) {  // equal P: the smaller key goes first
          if (ov >= 0 && ov < nphi) blocked |= Wk.key(C.slot[((u + du) << sh) + ov]).x < ckey;
        }
      }
      const unsigned ball = __ballot_sync(kFull, blocked);
      if (k < nc && (lane & 7) == 0 && !((ball >> (lane & 24)) & 0xffu)) {
        // two steps never share a slot: the lower bit is claimed first, so of
        // several that want the same ones, one gets both of its own
        const int bc = round_bit<SM>(c), bj = round_bit<SM>(jc);
        bool ok = care == 2;
        if (SM) pair = round_pair(Wk, c, jc);
        if (!ok && !(S.backs && round_held<SM>(c, jc, __uint_as_float(me)))) {
          ok = round_first(S.taken, min(bc, bj));
          if (ok && bc != bj) ok = round_first(S.taken, max(bc, bj));
        }
        const int i = ok ? atomicAdd(&S.n_fire, 1) : kRoundSteps;
        if (i < kRoundSteps) {
          const RoundStep st = round_step<SM>(c, j, pair, S.X.inv_r2);
          c = st.c;
          j = st.j;
          const RoundTime te = st.t;
          const double key = st.key, wc = pair.wc, wj = pair.wj;
          const double thr_c = st.chained && !st.from_j ? key : te.M;
          const double thr_j = st.chained && st.from_j ? key : te.M;
          // the promotions of c and j come later
          const bool late = j >= 0 && (wc <= thr_c || wj <= thr_j);
          if (late && care != 2) S.conflict[0] = 1;
          S.new_u[i] = late;
          S.c[i] = c;
          S.j[i] = j;
          S.key[i] = key;
          S.M[i] = te.M;
          S.l[i] = te.l;
          S.depth[i] = te.depth;
          S.thr_c[i] = thr_c;
          S.thr_j[i] = thr_j;
          const int jn = j >= 0 ? j : c;
          S.tile_c[i] = Wk.tile(c);
          S.tile_j[i] = Wk.tile(jn);
          S.xy_c[i] = Wk.xy(c);
          S.xy_j[i] = Wk.xy(jn);
          S.wlo[i] = make_float2(round_wlo(Wk.wlo(c)), round_wlo(Wk.wlo(jn)));
        }
      }
      __syncwarp();
    }
    __syncthreads();
    if (care == 2) {
      if (tid == 0) round_earliest<SM>();
      __syncthreads();
    }
    const int F = min(S.n_fire, kRoundSteps);
    if (!F || S.conflict[0]) {  // (F = 0: cannot happen)
      if (tid == 0) S.conflict[1] = 1;
      break;
    }
    FJG_PH(mark(kPhRRange); ++ph[kPhRRounds - kPhRSetup]; ph[kPhRSteps - kPhRSetup] += F; ph[kPhRCands - kPhRSetup] += nc;)
    // lanes per step: few steps, a warp each
    const int G = SM && F > W ? 8 : 32;

    // B: kinematics of the new jets, a lane per step
#pragma unroll 1
    for (int role = warp; role < 4; role += W) {
      FJG_PH(const long long q0 = clock64();)
      const int i = lane;
      const bool have = i < F;
      const int c = have ? S.c[i] : 0, j = have ? S.j[i] : -1;
      if (role == 2) {
        // weight, record, and the dead of the step
        int tile_c = 0, tile_j = 0, b = 0;
        float4 dc{}, dj{};
        float m_hi = 0.0f;
        if (have) {
          b = max(c, j);
          m_hi = __double2float_ru(S.M[i]);
          const float2 gc = S.xy_c[i];
          dc = make_float4(gc.x, gc.y, S.wlo[i].x, __double2float_ru(S.thr_c[i]));
          const int2 tpc = make_int2(S.tile_c[i], Wk.at(c));
          tile_c = tpc.x;
          S.tp_b[i] = tpc;
          if (j >= 0) {
            const float2 gj = S.xy_j[i];
            dj = make_float4(gj.x, gj.y, S.wlo[i].y, __double2float_ru(S.thr_j[i]));
            const int2 tpj = make_int2(S.tile_j[i], Wk.at(j));
            tile_j = tpj.x;
            S.tp_b[i] = c > j ? tpc : tpj;
            S.tp_a[i] = c > j ? tpj : tpc;
            const double w =
                fjk_weight(__dadd_rn(Wk.p4(0, c), Wk.p4(0, j)), __dadd_rn(Wk.p4(1, c), Wk.p4(1, j)), algo);
            S.w[i] = w;
            if (round_refuses(w)) S.conflict[1] = S.hopeless = 1;
          }
          RoundRec r;
          r.M = S.M[i];
          r.d = S.key[i];
          r.l = S.l[i];
          r.depth = S.depth[i];
          r.a = j >= 0 ? min(c, j) : -1;
          r.round = round;
          Wk.rec(b) = r;
        }
        __syncwarp();
#pragma unroll 1
        for (int q = 0; q < 2; ++q)
          round_bury<SM>(have && (!q || j >= 0), q ? tile_j : tile_c, 2 * b + q, q ? dj : dc, m_hi,
                         have ? S.l[i] : 0);
      } else if (role == 3) {
        if (have && j >= 0) {  // slot a as it was, to take the step back
          RoundDead& D = Wk.dead[max(c, j)];
          const RoundSlot& a = Wk.slots[min(c, j)];
#pragma unroll
          for (int q = 0; q < 4; ++q) D.p[q] = a.p[q];
          D.w = a.w;
          D.tm = a.tm;
          D.tl = a.tl;
          D.pos = a.pos;
        }
      } else if (have && j >= 0) {
        const double px = __dadd_rn(Wk.p4(0, c), Wk.p4(0, j)), py = __dadd_rn(Wk.p4(1, c), Wk.p4(1, j));
        if (role == 0) {
          const double phi = fjk_phi(px, py);
          S.phi[i] = phi;
          S.new_v[i] = round_v(S, phi);
        } else {
          const double pz = __dadd_rn(Wk.p4(2, c), Wk.p4(2, j)), E = __dadd_rn(Wk.p4(3, c), Wk.p4(3, j));
          const double rap = fjk_rap(px, py, pz, E);
          if (round_refuses_rap(rap)) S.conflict[1] = S.hopeless = 1;
          S.p4[0][i] = px;
          S.p4[1][i] = py;
          S.p4[2][i] = pz;
          S.p4[3][i] = E;
          S.rap[i] = rap;
          S.new_u[i] = round_u(S, rap);
        }
      }
      __syncwarp();
      FJG_PH(if (lane == 0 && A.phase && role < 3) atomicAdd(A.phase + kPhRRole0 + role, (unsigned long long)(clock64() - q0));)
    }
    // D1 and the targets
    FJG_PH(const long long qb = clock64();)
    round_phase_b(C, F, G, G == 32 ? max(1, (SM ? W - 3 : 2 * (W - 3)) / F) : 1);
    FJG_PH(if (tid == T - 32 && A.phase) atomicAdd(A.phase + kPhRScan, (unsigned long long)(clock64() - qb));)
    __syncthreads();
    FJG_PH(mark(kPhRB);)

    // C: the new state, a lane per step
    if (warp == 0) {
      if (lane < F) {
        const int i = lane;
        const int c = S.c[i], j = S.j[i];
        const int b = max(c, j);
        const int2 tb = S.tp_b[i];
        Wk.members[C.start[tb.x] + tb.y] = (Idx)kNone;
        Wk.tile(b) = (Idx)kNone;
        round_dirty(S, tb.x);
        if (j >= 0) {
          const int a = min(c, j);
          const int2 ta = S.tp_a[i];
          const int t = (S.new_u[i] << sh) + S.new_v[i];
          if (ta.x != tb.x) round_dirty(S, ta.x);
          if (t != ta.x) {
            Wk.members[C.start[ta.x] + ta.y] = (Idx)kNone;
            const int p = atomicAdd(&C.count[t], 1);
            if (C.start[t] + p < C.start[t + 1])
              Wk.place(C.start[t] + p, a, make_float2(__double2float_rn(S.rap[i]), __double2float_rn(S.phi[i])));
            else
              S.overflow = 1;
            Wk.tile(a) = (Idx)t;
            Wk.at(a) = (Idx)p;
          } else if (!SM) {
            Wk.place(C.start[t] + ta.y, a, make_float2(__double2float_rn(S.rap[i]), __double2float_rn(S.phi[i])));
          }
        }
      }
      if (lane == 0) {
        S.n_cand = 0;
        S.p_min = kRoundNone;
        S.task[0] = 0;
      }
    } else if (warp == 1) {
      if (lane < F && S.j[lane] >= 0) {
        const int i = lane;
        const int a = min(S.c[i], S.j[i]);
        const double rap = S.rap[i], phi = S.phi[i], w = S.w[i];
#pragma unroll
        for (int q = 0; q < 4; ++q) Wk.p4(q, a) = S.p4[q][i];
        Wk.w(a) = w;
        Wk.pos(a) = make_double2(rap, phi);
        Wk.xy(a) = make_float2(__double2float_rn(rap), __double2float_rn(phi));
        Wk.nhi(a) = inf;
        Wk.wlo(a) = round_weight(w);
        Wk.tlo(a) = fmaxf(__double2float_rd(S.M[i]), 0.0f);
        Wk.tm(a) = S.M[i];
        Wk.tl(a) = make_int2(S.l[i], S.depth[i]);
        Wk.nn(a) = (Idx)(Ws_::kNoSlot | Ws_::kTarget);  // its own group searches its neighbour
      }
    }
    __syncthreads();
    if (S.conflict[1]) break;
    n -= F;
    if (S.overflow) {  // a list is full: all lists again
      round_lists<SM>(n);
      if (tid == 0) S.overflow = 0;
      FJG_PH(++ph[kPhROverflows - kPhRSetup];)
    }
    FJG_PH(mark(kPhRC);)

    // D: each new jet against its window; the targets' searches (one may have
    // been taken by another step); the dead of each new jet's window (D2).  A
    // warp takes 32 / G of a kind at a time, or a part of one.
    const int ntg = min(S.n_targets, kRoundMaxTargets);
    __syncthreads();  // D adds targets
    const int per = 32 / G;
    const int parts = !SM && F + ntg <= kRoundSplit ? max(1, min(kRoundParts, W / (F + ntg))) : 1;
    // (parts of the targets' searches)
    const int pt = !SM && n >= kRoundCrowded * nt && nphi >= 5 ? 0 : parts, pts = pt ? pt : 1;
    const int uf = (F + per - 1) / per * parts, ut = (ntg + per - 1) / per * pts, ud = (F + per - 1) / per;
#pragma unroll 1
    for (;;) {
      int u = 0;
      if (lane == 0) u = atomicAdd(&S.task[1], 1);
      u = __shfl_sync(kFull, u, 0);
      if (u >= uf + ut + ud) break;
      FJG_PH(const long long qd = clock64();)
      const int q = G == 32 ? 0 : lane / 8;
      if (u < uf) {
        const int i = per * (u / parts) + q;
        round_new_jet(C, i < F && S.j[i < F ? i : 0] >= 0, i < F ? i : 0, G, u % parts, parts);
      } else if (u < uf + ut) {
        const int k = per * ((u - uf) / pts) + q;
        const int t = S.targets[k < ntg ? k : 0];
        round_search<SM>(k < ntg && (int)Wk.tile(t) != kNone, t, G, F + k, (u - uf) % pts, pt);
      } else {
        const int i = per * (u - uf - ut) + q;
        if (i < F && S.j[i] >= 0) {
          const double M = S.M[i];
          const float m_lo = __double2float_rd(M);
          const int tile = (S.new_u[i] << sh) + S.new_v[i];
          const RoundBox b = round_box(S, tile, tile);
          const int nb = b.nu * b.nv;
          bool bad = false;
#pragma unroll 1
          for (int k = lane & (G - 1); k < nb; k += G) {
            const int t = box_tile(S, b, k);
            const int x = C.head[t];
            if (x >= 0 && C.head_m[t] >= m_lo) bad |= round_d2<SM>(x, min(S.c[i], S.j[i]), M, S.l[i], S.depth[i]);
          }
          if (bad) S.conflict[2] = 1;
        }
        __syncwarp();
      }
      FJG_PH(if (lane == 0 && A.phase) atomicAdd(A.phase + (u < uf ? kPhRNewJet : u < uf + ut ? kPhRSearch : kPhRDead), (unsigned long long)(clock64() - qd));)
    }
    __syncthreads();
    const int ntg2 = S.n_targets;
    FJG_PH(mark(kPhRD); ph[kPhRTargets - kPhRSetup] += ntg2;)
    // (more targets than listed: only degenerate inputs)
    if (S.conflict[2] || ntg2 > kRoundMaxTargets) {
      if (tid == 0) S.conflict[0] = 1;
      break;
    }
    if (ntg2 > ntg) {  // slots that two new jets wanted
#pragma unroll 1
      for (int k = ntg + warp; k < ntg2; k += W) round_search<SM>(true, S.targets[k], 32, 0, 0, 1);
      __syncthreads();
    }
    FJG_PH(mark(kPhRE);)

    // F: the target bits off; changed tiles
    if (tid < ntg2 || (tid < F && S.j[tid] >= 0)) {
      if (tid < ntg2) Wk.nn(S.targets[tid]) &= (Idx)~Ws_::kTarget;
      if (tid < F && S.j[tid] >= 0) Wk.nn(min(S.c[tid], S.j[tid])) &= (Idx)~Ws_::kTarget;
    }
    const int nd = S.n_dirty, ndt = nd <= kRoundMaxDirty ? nd : nt;
    if (dense) {
#pragma unroll 1
      for (int k = warp; k < ndt; k += W) round_summary_warp<SM>(nd <= kRoundMaxDirty ? S.dirty[k] : k);
    } else {
#pragma unroll 1
      for (int k = tid; k < ndt; k += T) round_summary_thread<SM>(nd <= kRoundMaxDirty ? S.dirty[k] : k);
    }
    for (int k = tid; k < kRoundMaxTiles / 32; k += T) S.dirty_bits[k] = 0;
    __syncthreads();
    FJG_PH(mark(kPhRF);)
    if (tid == 0) {
      S.n_dirty = S.n_targets = S.n_fire = 0;
      S.task[1] = 0;
    }
    // (the next writers of these follow the next barriers)
  }
  __syncthreads();
  if (!(S.conflict[0] | S.conflict[1] | S.conflict[2])) break;
  // back to before the steps that came too early (D1, and D2 within a round: this
  // round's), and from there with more care
  round_line<SM>();
  const int r0 = min(S.back, round);
  const bool again = round < S.care_until;
  const int care = !S.conflict[2] ? 2 : !again ? 0 : round - r0 <= 4 * kRoundCareRounds ? 2 : 1;
  const bool hopeless = S.hopeless || S.backs >= kRoundMaxBacks + N / 2048 || (again && S.care == 2 && r0 == round);
  FJG_PH(ph[kPhRBacks - kPhRSetup] += 1; if (A.phase && tid == 0) {
    atomicAdd(A.phase + kPhRRetries, (unsigned long long)hopeless);
    for (int k = 0; k < 3; ++k) atomicAdd(A.phase + kPhRConflictA + k, (unsigned long long)(S.conflict[k] != 0));
    atomicAdd(A.phase + kPhRUndone, (unsigned long long)(round - r0));
  })
  __syncthreads();
  if (hopeless) return false;
  round_undo<SM>(r0);
  if (tid == 0) {
    ++S.backs;
    S.care = care;
    S.care_until = round + (care < 2 ? 2 * (round - r0) + kRoundCareRounds : max(S.alive - n, 0) + kRoundCareRounds / 4);
  }
  n = S.alive;
  ++round;
  FJG_PH(mark(kPhRSetup);)
  }

  // ---- records in sequential order
  Idx* order = Wk.members;
  int n2 = 1;
  while (n2 < N) n2 <<= 1;
  if constexpr (SM)
    round_sort_smem(C, N, n2, order);
  else
    round_sort(C, N, n2, order);
  FJG_PH(mark(kPhRSort);)
  // ---- outputs
  int jets = 0;
#pragma unroll 1
  for (int base = 0; base < N; base += T) {
    const int r = base + tid;
    const int s = r < N ? (int)order[r] : -1;
    RoundRec rec{};
    if (s >= 0) rec = Wk.rec(s);
    const bool jet = s >= 0 && rec.a < 0;
    const unsigned ball = __ballot_sync(kFull, jet);
    if (lane == 0) S.scan_tmp[warp] = __popc(ball);
    __syncthreads();
    int pre = 0, total = 0;
    for (int k = 0; k < W; ++k) {
      if (k < warp) pre += S.scan_tmp[k];
      total += S.scan_tmp[k];
    }
    if (s >= 0) {
      if (A.history) A.history[off + r] = jet ? StepRec{s, -1, rec.d} : StepRec{rec.a, s, rec.d};
      int par = rec.a;
      if (jet) {
        const int k = jets + pre + __popc(ball & ((1u << lane) - 1));
        double* jo = A.jets + (off + k) * 4;
        jo[0] = Wk.p4(0, s);
        jo[1] = Wk.p4(1, s);
        jo[2] = Wk.p4(2, s);
        jo[3] = Wk.p4(3, s);
        A.jet_label[off + k] = s;
        par = -(k + 1);
      }
      Wk.slots[s].parent = par;
    }
    jets += total;
    __syncthreads();
  }
  if (tid == 0) A.n_jets[e] = jets;
  if (A.owner) {
#pragma unroll 1
    for (int s = tid; s < N; s += T) {
      int v = Wk.slots[s].parent;
#pragma unroll 1
      for (int guard = 0; v >= 0 && guard < N; ++guard) v = Wk.slots[v].parent;
      A.owner[off + s] = v < 0 ? -v - 1 : -1;
    }
  }
  __syncthreads();
  FJG_PH(mark(kPhROut); ph[kPhREvents - kPhRSetup] = 1;
         if (A.phase && tid == 0) for (int k = kPhRSetup; k < kPhSlots; ++k)
           atomicAdd(A.phase + k, (unsigned long long)ph[k - kPhRSetup]);)
  return true;
}

}  // namespace fjg
