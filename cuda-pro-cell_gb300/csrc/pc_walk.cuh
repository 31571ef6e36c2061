// The tree walk: a whole run of the proliferation path in one launch, without level buffers.
//
// The level sweeps (pc_sweeps.cuh) write every dividing cell to HBM once per generation and
// compute both daughters' FP64 due times, and their rate is set by instruction issue and by
// the FP64 pipe (2 lanes per clock per SM), which alone allows 1.3e11 divisions/s. Here each
// warp walks trees depth-first instead: it keeps a stack of dividing cells in shared memory,
// pops 32 at a time, draws both daughters of each and pushes those that divide again, so a
// cell never leaves the SM, no generation waits for another, and the deepest stack is bounded
// by 32 cells per generation. A cell carries no absolute due time but the time left,
// rem = t_max - due, in FP32, and its sign decides leaf or division:
//
//   Filtered predicate. |rem - (t_max - due)| is bounded over the whole lineage by `band`
//   (host_walk_type in pc_api.cpp derives it), so whenever |rem| > band the sign is that of
//   the exact FP64 due time the level sweeps compare. A daughter with |rem| <= band (about 1
//   in 20000), like one whose first-attempt normal is rejected or not certainly inside the
//   truncation tau > 0, is parked and settled 32 at a time: its normal by the generic
//   sampler and, still inside the band, its due time by replaying its lineage from the initial
//   cell in FP64 with the operations of the sweeps. Counts are therefore bit-identical, and
//   the FP64 pipe does nothing for the other 99.99%.
//
// Leaves are never counted one by one: the daughters born at generation g of a histogram
// class are twice the cells that divided at g - 1, so leaves(g) = 2 D(g - 1) - D(g) - V(g)
// with D the cells that divide and V those that vanish at the phi cap. A popped cell adds 1
// to its class's D(g) in a per-warp window of shared memory (kCols classes x 32 generations);
// the window is flushed into the global table when its columns run out or the work ends.
//
// Load balance. Warps take initial cells from a global counter. A warp that is still walking
// while a quarter of all warps have nothing to do (or any, for long) writes its stack to its
// slot of a global buffer and stops; after a grid barrier those cells are dealt out evenly to
// all warps in another round, until none are left. A few initial cells with deep trees spread
// over the whole chip this way in three or four rounds, and no warp waits long for another.
//
// What bounds it (GB300, 2070 MHz; 32 divisions of a warp are one step): a step is about 115
// instructions, 57 of them on the ALU pipe (28 of 50 cycles per SM), 20 wide multiplies of Philox
// (23 cycles alone) and 33 shared-memory wavefronts, half of those the ziggurat's random lookups;
// measured alone it takes 50 cycles of an SM, 5.0 ps per division, and adding warps (24 to 32 per
// SM) changes that by 4%. A whole run of 2.27e9 divisions takes 13.1 ms, 5.8 ps per division,
// against 10.1 ps for the level sweeps; a run of 14e6 divisions of 1e6 initial cells 0.19 ms
// against 0.45 ms; 16 thousand divisions 0.033 ms against 0.16 ms and nine host round trips.
// 24 warps per SM with stacks of 400 cells, because a spill of 32 cells and their return cost
// about 350 instructions: 32 warps and 264 cells 14.0 ms, 28 and 320 13.2, 24 and 400 13.1, 20
// and 496 13.5. Cells kept as two 8-byte halves and type data 16 bytes apart: 33 wavefronts per
// step instead of 44 with 16-byte cells and the types inside the 128-byte columns.
#pragma once

#include "pc_sweeps.cuh"

namespace pc {

namespace {

constexpr int kWalkThreads = 768;
constexpr int kWalkWarps = kWalkThreads / 32;
constexpr int kWalkBlocksPerSm = 1;
constexpr uint32_t kCols = kWalkCols;   // histogram classes in a warp's window
// Shared-memory stack entries of a warp, parked ones included, and the cells a full step may start
// with: it pops 32 and adds at most 128, with up to 31 parked before it. 80 cells fewer leave 32 KB
// more of L1 to the lookups of initial cells and the local memory of the code around the steps, 80
// more save spills where trees are deep; which is worth more depends on the run, not on its form.
// 320 and 400 cells, ms: batches of 256 x 1e5 cells (4 divisions each) 1.34 and 1.53, 10 x 1e5 (12)
// 0.168 and 0.171, 4 x 25000 (270) 0.344 and 0.364, 256 x 1e4 (230) 4.24 and 4.21, 16 x 6.4e5 (210)
// 13.63 and 13.49; plain runs of 1e7 cells (4) 0.536 and 0.562, 1e6 (13) 0.158 and 0.167, 1e5 (240)
// 0.302 and 0.322, 1e7 (240) 14.26 and 14.00. Each kernel has the one that its largest loads want:
// a batch is most often many shallow runs, the longest plain runs are deep.
template <bool Batched>
constexpr uint32_t kStackCap = Batched ? 320 : 400;
template <bool Batched>
constexpr uint32_t kStackRoom = kStackCap<Batched> - 96u - 31u;
constexpr uint32_t kFirstPoll = 8;      // steps of a round before the first look at the idle warps
constexpr uint32_t kPollSteps = 32;     // steps between two looks at the number of idle warps
constexpr uint32_t kIdlePolls = 120;    // looks that found any idle warp after which cells are handed over
constexpr uint32_t kShortPolls = 6;     // ... that found a quarter of the warps idle
constexpr uint32_t kLongStack = 48;     // ... a quarter idle, one look, with at least so many cells

// A warp's window holds kCols histogram classes ("columns"): word `left` of a column counts the
// cells that divided with `left` = phi cap - g generations to go (D), word 0 the cells that
// vanished at the cap (V). The odd column stride spreads equal generations over the banks.
//
// A cell on the stack: the FP32 time left until t_max, its heap node, its initial cell (index
// within the instance) and meta = shared-memory address of its D counter | left << 18 |
// column << 28: one mask, one shift-add and one mask lead to its counter, its type and the phi
// cap's test, and a daughter's meta is its parent's minus kMetaChild. (Cells in global memory
// hold the address relative to the window.)
constexpr uint32_t kNoBin = ~0u;  // the next initial cell's bin is not known yet
constexpr uint32_t kColWords = 33;
constexpr uint32_t kMetaAddress = 0x3FFFCu;
constexpr uint32_t kMetaLeftShift = 18, kMetaColShift = 28;
constexpr uint32_t kMetaLeft = 31u << kMetaLeftShift;    // nonzero: the cell may divide
constexpr uint32_t kMetaDeeper = 30u << kMetaLeftShift;  // nonzero: its daughters may
constexpr uint32_t kMetaChild = 4u + (1u << kMetaLeftShift);
static_assert(kWalkMaxGen < kColWords && kCols <= 16, "one word per generation to go; four bits of column");

template <bool Batched>
struct alignas(16) WalkWarp {
  float4 rec[kCols];  // mean, sd, eps, band of the column's type
  uint2 key[kCols];   // its instance's seed
  uint2 aux[kCols];   // class; type index | phi cap << 16 | countable at g = 0 << 24
  uint32_t window[kCols * kColWords];
  // the stack: cells from the bottom, parked daughters from the top; two arrays, so that a
  // step's two daughters share the registers of their second half
  uint2 stack_t[kStackCap<Batched>];  // time left, node
  uint2 stack_m[kStackCap<Batched>];  // initial cell, meta
  // the round's state, out of the step's registers (uniform over the warp, written by lane 0)
  unsigned long long cpos, cend;                      // current range of initial cells
  unsigned long long divisions, vanished, uncounted;  // totals of the round so far
  uint32_t ncols, nspill, steps, recent, polls, max_gen, blocked, more, bin;
  uint32_t lpos, lend;  // current range of the cells handed over
  uint32_t taken, pad;  // supplies taken (0: none yet)
};

template <bool Batched>
struct alignas(16) WalkSmem {
  uint2 zig[kZigLayers];  // strip-test bound and scale of each ziggurat layer
  WalkWarp<Batched> warp[kWalkWarps];
  uint32_t finished;  // warps of the block that have finished the round
  uint32_t pad[3];
  WalkArgs w;  // the launch's arguments, for the code outside the step
};
static_assert(sizeof(WalkArgs) % 4 == 0, "copied word by word");

// Shared memory by address (walk cells carry addresses).
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <class T>
__device__ __forceinline__ T* shared_at(uint32_t address) {
  return static_cast<T*>(__cvta_shared_to_generic((size_t)address));
}

extern __shared__ __align__(16) unsigned char walk_smem[];
template <bool Batched>
__device__ __forceinline__ WalkSmem<Batched>& walk_shared() {
  return *reinterpret_cast<WalkSmem<Batched>*>(walk_smem);
}
template <bool Batched>
__device__ __forceinline__ WalkWarp<Batched>& walk_warp() {
  return walk_shared<Batched>().warp[threadIdx.x >> 5];
}

// The exact due time of a node, by its lineage from the initial cell: the operations of
// root_body and divide_body (pc_sweeps.cuh), in their order.
__device__ __noinline__ double replay_due(uint32_t node, uint32_t root, double mu, double sigma, float zlo, float zhi,
                                          uint32_t k0, uint32_t k1, const ZigTables& Z, uint32_t* error) {
  const u32x4 R = philox(u32x4{0u, 0u, root, kPurposeRoot}, k0, k1);
  const double u_age = unit53_open_closed(R.z, R.w);
  const u32x4 P0 = philox(u32x4{0u, 0u, root, kPurposePair}, k0, k1);
  const float z1 = draw_z(P0.y, pair_layer(P0, 1u), pair_wedge_bits(P0, 1u), 1ull, root, k0, k1, zlo, zhi, Z, error);
  const double tau1 = fma(sigma, widen_scaled(z1), mu);
  double due = tau1 * u_age + tau1;
  for (int s = 30 - __clz((int)node); s >= 0; --s) {
    const uint32_t n = node >> s, c = n & 1u;
    const u32x4 P = philox(u32x4{n >> 1, 0u, root, kPurposePair}, k0, k1);
    const float z = draw_z(c ? P.y : P.x, pair_layer(P, c), pair_wedge_bits(P, c), n, root, k0, k1, zlo, zhi, Z, error);
    due = due + fma(sigma, widen_scaled(z), mu);
  }
  return due;
}

template <bool Batched>
__device__ __forceinline__ const TypeDev& walk_type(const RunArgs& a, uint32_t ty) {
  if constexpr (Batched)
    return a.btypes[ty].t;
  else
    return a.types[ty];
}

// Checked build: a stack index in range (true at compile time otherwise).
template <bool Batched>
__device__ __forceinline__ bool stack_ok(uint32_t i) {
  return in_bounds(i < kStackCap<Batched>, walk_shared<Batched>().w.a.error);
}
template <bool Batched>
__device__ __forceinline__ uint4 stack_get(const WalkWarp<Batched>& W, uint32_t i) {
  if (!stack_ok<Batched>(i)) return make_uint4(0u, 0u, 0u, 0u);
  const uint2 t = W.stack_t[i], m = W.stack_m[i];
  return make_uint4(t.x, t.y, m.x, m.y);
}
template <bool Batched>
__device__ __forceinline__ void stack_put(WalkWarp<Batched>& W, uint32_t i, uint4 e) {
  if (!stack_ok<Batched>(i)) return;
  W.stack_t[i] = make_uint2(e.x, e.y);
  W.stack_m[i] = make_uint2(e.z, e.w);
}

// The warp's global region of a round: cells spilled, then handed over.
__device__ __forceinline__ uint4* walk_region(const WalkArgs& w, uint32_t round) {
  const uint32_t wid = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
  return w.region[round & 1u] + (uint64_t)wid * w.region_stride;
}

// The window into the global table: leaves(g) = 2 D(g - 1) - D(g) - (g == cap ? V : 0), in
// wrapping arithmetic (a cell handed over is counted by another warp than its parent). Lanes c
// and 16 + c take column c's even and odd generations. At most 2^30 cells are counted between two
// flushes, so 32 bits hold their sums.
// A window is flushed whenever the next initial cells bring a 17th class: every 20 to 60 cells where
// a bin has many types or few cells. One column after another, lanes as generations, took 45
// instructions each. 1.6e7 cells of 24 types, 1.25 divisions each: 2.23 -> 1.75 ms; 4e6 cells in
// bins of 8, 8 types 0.72 -> 0.58; 512 instances of 4096 cells and 24 types 0.63 -> 0.54.
template <bool Batched>
__device__ __noinline__ void walk_flush(uint32_t ncols) {
  const RunArgs& a = walk_shared<Batched>().w.a;
  WalkWarp<Batched>& W = walk_warp<Batched>();
  const uint32_t lane = threadIdx.x & 31u, c = lane & 15u;
  __syncwarp();
  const uint2 x = W.aux[c];
  const int cap = c < ncols ? (int)((x.y >> 16) & 0xFFu) : -1;
  const uint32_t last = (uint32_t)__reduce_max_sync(kFull, cap);
  uint32_t* const word = W.window + c * kColWords + cap;  // D(0); D(g) g words before it, V at g = cap
  uint32_t divisions = 0, vanished = 0, deepest = 0, before = 0;
  if (ncols != 0u)
    for (uint32_t g = lane >> 4; g <= last + (lane >> 4); g += 2u) {
      uint32_t d = 0, v = 0;
      if ((int)g <= cap) {
        d = word[-(int)g];
        word[-(int)g] = 0u;
        if ((int)g == cap) {
          v = d;
          d = 0;
        }
      }
      // D(g - 1): the odd lane's of the step before, the even lane's of this one
      const uint32_t above = __shfl_xor_sync(kFull, lane < 16u ? d : before, 16);
      before = d;
      const unsigned long long leaves = 2ull * above - d - v;
      if (g != 0u && leaves != 0ull && in_bounds(g < a.hist_gens && x.x < a.nclass, a.error))
        atomicAdd(a.hist + (uint64_t)g * a.nclass + x.x, leaves);
      divisions += d;
      vanished += v;
      if (d != 0u) deepest = g + 1u;
    }
  divisions = __reduce_add_sync(kFull, divisions);
  vanished = __reduce_add_sync(kFull, vanished);
  deepest = __reduce_max_sync(kFull, deepest);
  if (lane == 0u) {
    W.divisions += divisions;
    W.vanished += vanished;
    W.max_gen = max(W.max_gen, deepest);
  }
  __syncwarp();
}

// The 32 bottom cells of a full stack of `n` cells to the warp's global region.
template <bool Batched>
__device__ __forceinline__ void walk_spill(const WalkArgs& w, WalkWarp<Batched>& W, uint32_t round, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nspill = W.nspill;
  uint4 low = stack_get(W, lane);
  low.w -= shared_address(W.window);
  __syncwarp();
  if (nspill + 32u <= w.region_stride) {
    __stcg(walk_region(w, round) + nspill + lane, low);
    if (lane == 0u) W.nspill = nspill + 32u;
  } else if (lane == 0u) {
    atomicOr(w.a.error, kErrWalkStack);  // the run's counts are discarded
  }
  for (uint32_t i = 32u; i < n; i += 32u) {
    uint4 x = make_uint4(0u, 0u, 0u, 0u);
    if (i + lane < n) x = stack_get(W, i + lane);
    __syncwarp();
    if (i + lane < n) stack_put(W, i + lane - 32u, x);
    __syncwarp();
  }
}

// One step: up to 32 dividing cells off the stack (Full: exactly 32), both daughters of each.
// Returns whether daughters were parked.
template <bool Batched, bool Full>
__device__ __forceinline__ bool walk_step(const uint32_t* ks, const WalkSmem<Batched>& S, WalkWarp<Batched>& W, uint32_t lane,
                                          uint32_t lt, uint32_t& sp, uint32_t& np) {
  const uint32_t n = Full ? 32u : min(sp, 32u);
  const uint32_t base = sp - n;
  const bool act = Full || lane < n;
  const uint2 et = W.stack_t[base + lane], em = W.stack_m[base + lane];
  const uint32_t node = et.y, root = em.x;
  const uint32_t meta = act ? em.y : 0u;  // a lane without a cell reads column 0's type
  if (act) atomicAdd(shared_at<uint32_t>(meta & kMetaAddress), 1u);
  const float4 t = *shared_at<const float4>(shared_address(W.rec) + (meta >> (kMetaColShift - 4u)));
  u32x4 P;
  if constexpr (Batched) {
    const uint2 key = *shared_at<const uint2>(shared_address(W.key) + (meta >> (kMetaColShift - 3u)));
    P = philox(u32x4{node, 0u, root, kPurposePair}, key.x, key.y);
  } else {
    P = philox_ks(u32x4{node, 0u, root, kPurposePair}, ks);
  }
  const uint2 q0 = S.zig[pair_layer(P, 0u)], q1 = S.zig[pair_layer(P, 1u)];
  const uint32_t m0 = P.x & 0x7FFFFFFFu, m1 = P.y & 0x7FFFFFFFu;
  const float z0 = __uint_as_float(__float_as_uint(__fmul_rn((float)m0, __uint_as_float(q0.y))) ^ (P.x & 0x80000000u));
  const float z1 = __uint_as_float(__float_as_uint(__fmul_rn((float)m1, __uint_as_float(q1.y))) ^ (P.y & 0x80000000u));
  const float t0 = __fmaf_rn(t.y, z0, t.x), t1 = __fmaf_rn(t.y, z1, t.x);
  const float rem = __uint_as_float(et.x);
  const float r0 = __fsub_rn(rem, t0), r1 = __fsub_rn(rem, t1);
  // settled: strip test, certainly tau > 0, the time left certainly of its sign
  const bool ok0 = (m0 < q0.x) & (t0 > t.z) & (fabsf(r0) > t.w);
  const bool ok1 = (m1 < q1.x) & (t1 > t.z) & (fabsf(r1) > t.w);
  // a daughter in time goes on the stack, unless the phi cap keeps it from dividing
  const bool deeper = (meta & kMetaDeeper) != 0u;
  const float least = deeper ? 0.0f : INFINITY;
  const bool go0 = act & ok0 & (r0 > least), go1 = act & ok1 & (r1 > least);
  const uint32_t b0 = __ballot_sync(kFull, go0), b1 = __ballot_sync(kFull, go1);
  if (!deeper & act) {
    const uint32_t v = (ok0 & (r0 > 0.0f) ? 1u : 0u) + (ok1 & (r1 > 0.0f) ? 1u : 0u);
    if (v != 0u) atomicAdd(W.window + (meta >> kMetaColShift) * kColWords, v);
  }
  const uint32_t c0 = __popc(b0);
  const uint2 child = make_uint2(root, meta - kMetaChild);
  if (go0) {
    const uint32_t at = base + __popc(b0 & lt);
    if (stack_ok<Batched>(at)) {
      W.stack_t[at] = make_uint2(__float_as_uint(r0), 2u * node);
      W.stack_m[at] = child;
    }
  }
  if (go1) {
    const uint32_t at = base + c0 + __popc(b1 & lt);
    if (stack_ok<Batched>(at)) {
      W.stack_t[at] = make_uint2(__float_as_uint(r1), 2u * node + 1u);
      W.stack_m[at] = child;
    }
  }
  sp = base + c0 + __popc(b1);
  const bool p0 = act & !ok0, p1 = act & !ok1;
  const bool parked = __any_sync(kFull, p0 | p1);
  if (parked) {
    const uint32_t k0 = __ballot_sync(kFull, p0), k1 = __ballot_sync(kFull, p1);
    const uint32_t at = kStackCap<Batched> - 1u - np - __popc(k0 & lt) - __popc(k1 & lt);
    if (p0) stack_put(W, at, make_uint4(et.x, 2u * node, child.x, child.y));
    if (p1) stack_put(W, at - (p0 ? 1u : 0u), make_uint4(et.x, 2u * node + 1u, child.x, child.y));
    np += __popc(k0) + __popc(k1);
  }
  __syncwarp();  // the pushes are visible to the next step
  return parked;
}

// The normal of a parked daughter. Its first attempt and the retry that follows a rejected
// wedge or a truncated timer (the first two words of the node's stream) settle all but about
// 1% of them, with every lane on the same instructions; the rest (tails, second rejections)
// go through the sampler's loop (slow_z), which gives the same value from the start.
template <bool Batched>
__device__ __forceinline__ float parked_z(const WalkSmem<Batched>& S, const RunArgs& a, uint32_t node, uint32_t root, uint2 key,
                                          float zlo, float zhi) {
  const uint32_t c = node & 1u;
  const u32x4 P = philox(u32x4{node >> 1, 0u, root, kPurposePair}, key.x, key.y);
  const uint32_t j = c ? P.y : P.x, layer = pair_layer(P, c), wedge = pair_wedge_bits(P, c);
  const uint2 q = S.zig[layer];
  const uint32_t mag = j & 0x7FFFFFFFu;
  const float x = __fmul_rn((float)mag, __uint_as_float(q.y));
  const float f0 = __ldg(&a.zig->f[layer]), f1 = __ldg(&a.zig->f[layer + 1u]);
  const float y = fadd(f0, fmul(unit_closed_open(wedge), fsub(f1, f0)));
  const bool tail = mag >= q.x && layer == 0u;
  bool ok = mag < q.x || (!tail && y < zig_expf(fmul(-0.5f, fmul(x, x))));
  float z = __uint_as_float(__float_as_uint(x) | (j & 0x80000000u));
  ok = ok && z >= zlo && z <= zhi;
  if (!ok && !tail) {
    const u32x4 B = philox(u32x4{node, 0u, root, kPurposeChild}, key.x, key.y);
    const uint2 r = S.zig[B.y & kZigLayerMask];
    const uint32_t m = B.x & 0x7FFFFFFFu;
    z = __uint_as_float(__float_as_uint(__fmul_rn((float)m, __uint_as_float(r.y))) | (B.x & 0x80000000u));
    ok = m < r.x && z >= zlo && z <= zhi;
  }
  if (!ok) z = slow_z(j, layer, wedge, node, root, key.x, key.y, zlo, zhi, *a.zig, a.error);
  return z;
}

// Settles up to 32 parked daughters; those that divide again go on the stack.
template <bool Batched>
__device__ __forceinline__ void walk_settle(const WalkSmem<Batched>& S, WalkWarp<Batched>& W, uint32_t lane,
                                            uint32_t lt, uint32_t& sp, uint32_t& np) {
  const RunArgs& a = S.w.a;
  const uint32_t n = min(np, 32u);
  bool emit = false;
  uint32_t vanished = 0, uncounted = 0;
  uint4 e = make_uint4(0u, 0u, 0u, 0u);
  if (lane < n) {
    e = stack_get(W, kStackCap<Batched> - np + lane);
    const uint32_t col = e.w >> kMetaColShift;
    const uint2 x = W.aux[col], key = W.key[col];
    const float4 t = W.rec[col];
    const TypeDev& T = walk_type<Batched>(a, x.y & 0xFFFFu);
    const float zlo = __ldg(&T.zlo), zhi = __ldg(&T.zhi);
    const bool initial = e.y == 1u;
    const double t_max = __ldg(&T.t_max);
    float left = __uint_as_float(e.x), tau = __fmaf_rn(t.y, parked_z(S, a, e.y, e.z, key, zlo, zhi), t.x);
    // An initial cell's e.x is 1 + U, and its time left is found as in walk_roots: replaying all of
    // them in FP64 (one in most batches of 32) cost more than the rest of the settling, 0.12 ms
    // of 2.03 for 25.6e6 initial cells against 0.04 of 1.86.
    if (initial) {
      tau = __fmul_rn(tau, left);
      left = (float)t_max;
    }
    float rem = __fsub_rn(left, tau);
    bool leaf = rem < 0.0f;
    if (!(fabsf(rem) > t.w)) {
      const double due =
          replay_due(e.y, e.z, __ldg(&T.mu), __ldg(&T.sigma), zlo, zhi, key.x, key.y, *a.zig, a.error);
      leaf = gt_nonneg(due, t_max);
      rem = (float)(t_max - due);
    }
    e.x = __float_as_uint(rem);
    if (!leaf && (e.w & kMetaLeft) != 0u) {
      emit = true;
    } else if (!leaf) {
      if (initial)
        vanished = 1u;
      else
        atomicAdd(W.window + col * kColWords, 1u);
    } else if (initial) {  // counted here: no D(g - 1) stands for it
      if (!(x.y & (1u << 24)))
        uncounted = 1u;
      else if (in_bounds(x.x < a.nclass, a.error))
        atomicAdd(a.hist + x.x, 1ull);
    }
  }
  const uint32_t em = __ballot_sync(kFull, emit);
  const uint32_t nv = __popc(__ballot_sync(kFull, vanished != 0u)), nu = __popc(__ballot_sync(kFull, uncounted != 0u));
  if (lane == 0u && (nv | nu) != 0u) {
    W.vanished += nv;
    W.uncounted += nu;
  }
  np -= n;
  if (emit) stack_put(W, sp + __popc(em & lt), e);
  sp += __popc(em);
  __syncwarp();
}

// The next up to `batch` initial cells of the warp's range: type, first timer, initial age;
// those that divide go on the stack, unsettled ones to the parked daughters.
template <bool Batched>
__device__ __forceinline__ void walk_roots(const WalkSmem<Batched>& S, WalkWarp<Batched>& W, uint32_t lane,
                                           uint32_t lt, uint32_t& sp, uint32_t& np) {
  const RunArgs& a = S.w.a;
  const uint64_t cpos = W.cpos, cend = W.cend;
  // bin of the first one: the one before continues, or by 32-way search the largest b with
  // bin_start[b] <= cpos
  uint32_t b0 = W.bin;
  if (b0 == kNoBin) {
    uint32_t span = a.nbins;  // b in [b0, b0 + span)
    b0 = 0;
    while (span > 1u) {
      const uint32_t step = (span + 31u) / 32u;
      const uint32_t le = __ballot_sync(kFull, lane * step < span && __ldg(a.bin_start + b0 + lane * step) <= cpos);
      const uint32_t k = 31u - (uint32_t)__clz((int)le);  // lane 0 always holds
      b0 += k * step;
      span = min(step, span - k * step);
    }
  }
  const uint32_t want = (uint32_t)min((unsigned long long)S.w.batch, (unsigned long long)(cend - cpos));
  const uint64_t rg = cpos + lane;
  // every bin holds a cell, so 32 consecutive cells span at most 32 bins; most often they are
  // all of the first one
  unsigned long long bound = __ldg(a.bin_start + b0 + 1u);
  uint32_t off = 0;  // bins whose end is <= rg
  if (cpos + want >= bound) {
    bound = __ldg(a.bin_start + min(b0 + 1u + lane, a.nbins));
#pragma unroll
    for (uint32_t s = 16u; s != 0u; s >>= 1) {
      const unsigned long long e = __shfl_sync(kFull, bound, (int)(off + s - 1u));
      if (e <= rg) off += s;
    }
  }
  bool act = lane < want;
  const uint32_t bin = min(b0 + off, a.nbins - 1u);
  const uint32_t next_bin = min(bin + (__shfl_sync(kFull, bound, (int)off) <= rg + 1u ? 1u : 0u), a.nbins - 1u);
  uint32_t type_begin = 0, ntypes = a.ntypes, fallback = a.fallback, k0 = a.k0, k1 = a.k1;
  uint64_t root_begin = 0;
  double t_max = a.t_max;
  if (Batched) {
    const InstanceDev& I = a.inst[__ldg(a.bin_inst + bin)];
    type_begin = I.type_begin;
    ntypes = I.ntypes;
    fallback = I.fallback;
    k0 = I.k0;
    k1 = I.k1;
    root_begin = I.root_begin;
    t_max = I.t_max;
  }
  const uint32_t root = (uint32_t)(rg - root_begin);
  const u32x4 Q = philox(u32x4{0u, 0u, root, kPurposeRoot}, k0, k1);
  // u < cumulative ratio on the 53-bit integers
  const unsigned long long m = ((unsigned long long)Q.x << 21) | (Q.y >> 11);
  // (the first type whose threshold is above m: thresholds need not ascend). Four at a time: a
  // batch's types rarely stay in L1, and 64 loads one after another set its time (4.2e6 cells of 64
  // instances with 64 types 1.35 -> 0.94 ms, the level sweeps 1.15; 1.6e7 plain cells 3.29 -> 2.76).
  auto threshold = [&](uint32_t i) { return __ldg(&walk_type<Batched>(a, type_begin + i).w_cum); };
  uint32_t ty = fallback, i = 0;
  bool chosen = false;
  for (; !chosen && i + 4u <= ntypes; i += 4u) {
    const unsigned long long b0 = threshold(i), b1 = threshold(i + 1u), b2 = threshold(i + 2u), b3 = threshold(i + 3u);
    chosen = m < b0 || m < b1 || m < b2 || m < b3;
    if (chosen) ty = i + (m < b0 ? 0u : m < b1 ? 1u : m < b2 ? 2u : 3u);
  }
  for (; !chosen && i < ntypes; ++i) {
    chosen = m < threshold(i);
    if (chosen) ty = i;
  }
  const uint32_t info = __ldg(a.bin_info + bin), cap = info & 0xFFu;
  const uint32_t cls = Batched ? __ldg(a.bin_class + bin) + ty : bin * a.ntypes + ty;
  const TypeDev& T = walk_type<Batched>(a, type_begin + ty);
  const float4 t = __ldg(reinterpret_cast<const float4*>(&T.w_mean));
  const float band = __fmaf_rn((float)cap, t.w, __ldg(&T.w_band));
  const bool quiescent = __ldg(&T.mode) == kModeQuiescent;
  const u32x4 P = philox(u32x4{0u, 0u, root, kPurposePair}, k0, k1);
  const uint2 zk = S.zig[pair_layer(P, 1u)];
  const uint32_t mag = P.y & 0x7FFFFFFFu;
  const float z =
      __uint_as_float(__float_as_uint(__fmul_rn((float)mag, __uint_as_float(zk.y))) ^ (P.y & 0x80000000u));
  const float tau = __fmaf_rn(t.y, z, t.x);
  // 1 + U with the first 24 bits of U, then the time left at the first division
  const float one_u = __fmaf_rn((float)(Q.z >> 8), 0x1p-24f, 1.0f);
  const float rem = __fsub_rn((float)t_max, __fmul_rn(tau, one_u));
  const bool sure = mag < zk.x && tau > t.z && fabsf(rem) > band;
  const bool leaf = quiescent || (sure && rem < 0.0f);
  const bool parked = !quiescent && !sure;
  // window columns: the columns there are by comparison, one after another, then one for each new
  // class, in the order of its first lane; lanes from the first class that finds none are put off.
  // (One class after another, as many turns as classes: 1.6e7 cells of 24 types, 1.25 divisions each,
  // 1.75 ms, now 1.45; 4e6 cells in bins of 8, 8 types 0.58, now 0.48; of one type that hardly
  // divide, whose turns were few, 0.33 and 0.35.)
  const bool need = act && (parked || (!leaf && cap != 0u));
  const uint32_t ncols0 = W.ncols;
  uint32_t col = 0, ncols = ncols0, limit = 32u;
  if (__any_sync(kFull, need)) {
    const uint32_t first = (uint32_t)__ffs((int)__match_any_sync(kFull, need ? cls : ~0u)) - 1u;
    const uint32_t mine = lane < ncols0 ? W.aux[lane].x : 0u;  // class of column `lane`
    bool found = false;
    for (uint32_t c = 0; c < ncols0; ++c)
      if (__shfl_sync(kFull, mine, (int)c) == cls) {
        col = c;
        found = true;
      }
    const bool fresh = need && !found && first == lane;
    const uint32_t nw = __ballot_sync(kFull, fresh);
    if (nw != 0u) {
      if (fresh) col = ncols0 + __popc(nw & lt);
      const uint32_t over = __ballot_sync(kFull, fresh && col >= kCols);
      if (over != 0u) limit = (uint32_t)__ffs((int)over) - 1u;
      if (fresh && col < kCols) {
        W.rec[col] = make_float4(t.x, t.y, t.z, band);
        W.key[col] = make_uint2(k0, k1);
        W.aux[col] = make_uint2(cls, (type_begin + ty) | (cap << 16) | ((info & 0x100u) << 16));
      }
      const uint32_t of_first = __shfl_sync(kFull, col, (int)first);
      if (!found) col = of_first;
      ncols = min(ncols0 + (uint32_t)__popc(nw), kCols);
    }
  }
  act = act && lane < limit;
  const bool emit = act && sure && !leaf && cap != 0u;
  const bool park = act && parked;
  const bool counted = (info & 0x100u) != 0u;
  const uint32_t nv = __popc(__ballot_sync(kFull, act && sure && !leaf && cap == 0u));
  const uint32_t nu = __popc(__ballot_sync(kFull, act && leaf && !counted));
  // One addition per class of the 32 cells. Neighbouring ranges are walked at the same time, so a
  // bin of thousands of cells is added to by dozens of warps at once; with one addition per run of
  // equal classes (count_leaves) 1.6e7 cells in 800 bins that mostly do not divide took 0.52 ms with
  // one type and 1.10 with two, whose runs are short; 0.33 and 0.35 so (the root sweep 0.38 and 0.41).
  const bool one = act && leaf && counted && in_bounds(cls < a.nclass, a.error);
  const uint32_t ones = __ballot_sync(kFull, one);
  if (ones != 0u) {
    const uint32_t same = __match_any_sync(kFull, cls) & ones;
    if (one && (same & lt) == 0u) atomicAdd(a.hist + cls, (unsigned long long)__popc(same));
  }
  const uint4 e = make_uint4(__float_as_uint(rem), 1u, root,
                             (shared_address(W.window) + 4u * (col * kColWords + cap)) | (cap << kMetaLeftShift) |
                                 (col << kMetaColShift));
  const uint32_t em = __ballot_sync(kFull, emit), pk = __ballot_sync(kFull, park);
  if (emit) stack_put(W, sp + __popc(em & lt), e);
  if (park) stack_put(W, kStackCap<Batched> - 1u - np - __popc(pk & lt), make_uint4(__float_as_uint(one_u), e.y, e.z, e.w));
  sp += __popc(em);
  np += __popc(pk);
  const uint32_t took = min(want, limit);
  const uint32_t bin_after = __shfl_sync(kFull, next_bin, (int)(took - 1u));
  if (lane == 0u) {
    W.vanished += nv;
    W.uncounted += nu;
    W.ncols = ncols;
    W.cpos = cpos + took;
    if (took != 0u) W.bin = bin_after;
    if (took < want) W.blocked = 1u;  // the window is full: walk what is here, then flush it
  }
  __syncwarp();
}

// Hands the warp's cells over to the next round: the stack after the spilled ones, the columns'
// types, and the initial cells it has taken but not begun.
template <bool Batched>
__device__ __noinline__ void walk_hand_over(uint32_t round, uint32_t sp) {
  const WalkArgs& w = walk_shared<Batched>().w;
  WalkWarp<Batched>& W = walk_warp<Batched>();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t wid = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
  const uint32_t nspill = W.nspill, ncols = W.ncols;
  WalkRound& R = w.ctl->round[round & 3u];
  uint4* const region = walk_region(w, round);
  for (uint32_t i = lane; i < sp; i += 32u)
    if (nspill + i < w.region_stride) {
      uint4 e = stack_get(W, i);
      e.w -= shared_address(W.window);
      __stcg(region + nspill + i, e);
    }
  uint4* cols = w.cols[round & 1u] + (uint64_t)wid * (kCols * 2u);
  if (lane < ncols) {
    const uint4 t = *reinterpret_cast<const uint4*>(W.rec + lane);
    const uint2 key = W.key[lane], x = W.aux[lane];
    __stcg(cols + 2u * lane, t);
    __stcg(cols + 2u * lane + 1u, make_uint4(key.x, key.y, x.x, x.y));
  }
  __threadfence();
  __syncwarp();
  if (lane == 0u) {
    const uint32_t n = min(nspill + sp, (uint32_t)w.region_stride);
    if (nspill + sp > n) atomicOr(w.a.error, kErrWalkStack);
    // sources in the order of their first cells
    const unsigned long long at = atomicAdd(&R.handed, (1ull << 32) | n);
    w.sources[round & 1u][at >> 32] = make_uint4(wid, n, ncols, (uint32_t)at);
    if (W.cpos < W.cend) {
      const uint32_t k = atomicAdd(&R.ranges, 1u);
      w.ranges[round & 1u][k] = make_ulonglong2(W.cpos, W.cend);
    }
  }
  walk_flush<Batched>(ncols);
}

// The warp's next supply: a range of initial cells (round 0, or part of one given back), or a
// range of the cells handed over, which it then loads from one source after another.
template <bool Batched>
__device__ __noinline__ void walk_supply(uint32_t round) {
  const WalkArgs& w = walk_shared<Batched>().w;
  WalkWarp<Batched>& W = walk_warp<Batched>();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nwarps = gridDim.x * kWalkWarps;
  WalkRound& R = w.ctl->round[round & 3u];
  uint32_t supplies, parts = 1, nparts = 0, per = 0;
  unsigned long long cells = 0;
  if (round == 0u) {
    supplies = (uint32_t)((w.root_hi - w.root_lo + w.chunk - 1u) / w.chunk);  // < 2^32 - warps (run_walk)
  } else {
    const WalkRound& prev = w.ctl->round[(round - 1u) & 3u];
    cells = __ldcg(&prev.handed) & 0xFFFFFFFFull;
    parts = (w.chunk + w.batch - 1u) / w.batch;  // of a range given back
    nparts = __ldcg(&prev.ranges) * parts;
    per = (uint32_t)min(32ull, (cells + nwarps - 1u) / nwarps);
    supplies = nparts + (uint32_t)((cells + per - 1u) / per);
  }
  // The number of this supply: the first one of each warp is its own (consecutive ones on
  // different SMs), the later ones come from the counter, read before it is advanced so that
  // thousands of warps that find nothing do not queue up at it.
  uint32_t k = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  if (W.taken != 0u) {
    k = supplies;
    if (lane == 0u && nwarps + __ldcg(&R.next) < supplies) k = nwarps + atomicAdd(&R.next, 1u);
    k = __shfl_sync(kFull, k, 0);
  }
  __syncwarp();
  if (lane == 0u) {
    W.taken = 1u;
    if (k >= supplies) {
      W.more = 0u;
    } else if (round == 0u) {
      W.cpos = w.root_lo + (unsigned long long)k * w.chunk;
      W.cend = min(W.cpos + w.chunk, (unsigned long long)w.root_hi);
      W.bin = kNoBin;
    } else if (k < nparts) {
      const ulonglong2 range = __ldcg(w.ranges[(round - 1u) & 1u] + k / parts);
      const unsigned long long at = range.x + (unsigned long long)(k % parts) * w.batch;
      if (at < range.y) {
        W.cpos = at;
        W.cend = min(at + w.batch, range.y);
        W.bin = kNoBin;
      }
    } else {
      W.lpos = (k - nparts) * per;
      W.lend = (uint32_t)min((unsigned long long)W.lpos + per, cells);
    }
  }
  __syncwarp();
}

// The next cells of the warp's range of cells handed over, those of one source, with the
// source's columns after the window's own. Returns the cells put on the stack (0: the window
// has no room for the columns).
template <bool Batched>
__device__ __noinline__ uint32_t walk_load(uint32_t round, uint32_t sp) {
  const WalkArgs& w = walk_shared<Batched>().w;
  WalkWarp<Batched>& W = walk_warp<Batched>();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t old = (round - 1u) & 1u;
  const uint32_t lpos = W.lpos, lend = W.lend, ncols = W.ncols;
  // the last source whose first cell is at most lpos, by 32-way search
  uint32_t src = 0, span = (uint32_t)(__ldcg(&w.ctl->round[(round - 1u) & 3u].handed) >> 32);
  while (span > 1u) {
    const uint32_t step = (span + 31u) / 32u;
    const uint32_t le =
        __ballot_sync(kFull, lane * step < span && __ldcg(&w.sources[old][src + lane * step].w) <= lpos);
    const uint32_t k = 31u - (uint32_t)__clz((int)le);
    src += k * step;
    span = min(step, span - k * step);
  }
  const uint4 h = __ldcg(w.sources[old] + src);  // warp, cells, columns, first cell
  if (ncols + h.z > kCols) {
    __syncwarp();
    if (lane == 0u) W.blocked = 1u;
    __syncwarp();
    return 0u;
  }
  const uint4* cols = w.cols[old] + (uint64_t)h.x * (kCols * 2u);
  if (lane < h.z) {
    const uint4 k = __ldcg(cols + 2u * lane + 1u);
    *reinterpret_cast<uint4*>(W.rec + ncols + lane) = __ldcg(cols + 2u * lane);
    W.key[ncols + lane] = make_uint2(k.x, k.y);
    W.aux[ncols + lane] = make_uint2(k.z, k.w);
  }
  const uint32_t n = min(lend, h.w + h.y) - lpos;  // at most 32
  if (lane < n) {
    // A stack's cells grow shallower, with larger trees, towards its bottom, so a supply takes
    // every m-th cell: the source's cells j, j + m, ... for j = 0, then 1, ... (32 neighbours
    // instead: 7.7e8 divisions of 256 instances 7.9 ms and 8 rounds against 6.5 and 6, 3.9e7
    // divisions of 1e5 initial cells 0.55 against 0.45 ms.)
    const uint32_t m = (h.y + 31u) / 32u, a = h.y / m, b = h.y % m;
    const uint32_t p = lpos - h.w + lane;
    const uint32_t j = p < b * (a + 1u) ? p / (a + 1u) : (p - b) / a;
    const uint32_t i = j + (p - j * a - min(j, b)) * m;
    uint4 e = __ldcg(w.region[old] + (uint64_t)h.x * w.region_stride + i);
    e.w += shared_address(W.window) + 4u * kColWords * ncols + (ncols << kMetaColShift);
    stack_put(W, sp + lane, e);
  }
  if (lane == 0u) {
    W.ncols = ncols + h.z;
    W.lpos = lpos + n;
  }
  __syncwarp();
  return n;
}

// Everything but full steps: settles parked daughters, refills the stack, walks partial steps,
// spills, hands over or flushes. Returns sp | np << 16 with 32 <= sp <= kStackRoom and np < 32,
// or kWalkDone.
constexpr uint32_t kWalkDone = ~0u;

template <bool Batched>
__device__ __noinline__ uint32_t walk_manage(const uint32_t round, uint32_t sp, uint32_t np, const uint32_t steps) {
  const WalkSmem<Batched>& S = walk_shared<Batched>();
  WalkWarp<Batched>& W = walk_warp<Batched>();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t recent = W.recent + steps;  // steps since the last look at the idle warps
  bool hand_over = false;
  for (;;) {
    __syncwarp();
    if (np >= 32u || (np != 0u && (hand_over || (sp == 0u && W.nspill == 0u && (!W.more || W.blocked))))) {
      walk_settle<Batched>(S, W, lane, lt, sp, np);
      continue;
    }
    if (recent >= kPollSteps && sp != 0u) {
      // Handing cells over costs a round (10 to 15 us, most of it latency), so a warp with a
      // short stack walks on for a while: it often ends within that time.
      const uint32_t idle = __shfl_sync(kFull, __ldcg(&S.w.ctl->round[round & 3u].idle), 0);
      const uint32_t polls =
          W.polls + (idle >= (gridDim.x * kWalkWarps) / 4u ? kIdlePolls / kShortPolls : idle != 0u ? 1u : 0u);
      const uint32_t walked = W.steps + recent;
      recent = 0;
      // (cells of another warp that this one has taken but not loaded are walked first)
      hand_over = W.lpos >= W.lend && (polls >= kIdlePolls || (polls >= kIdlePolls / kShortPolls &&
                                                               sp + W.nspill >= kLongStack));
      const bool full = walked >= (1u << 25);  // long before a 32-bit counter of the window wraps
      if (full) walk_flush<Batched>(W.ncols);
      __syncwarp();
      if (lane == 0u) {
        W.polls = polls;
        W.steps = full ? 0u : walked;
      }
      continue;
    }
    if (hand_over) {
      walk_hand_over<Batched>(round, sp);
      return kWalkDone;
    }
    if (sp > kStackRoom<Batched>) {
      walk_spill(S.w, W, round, sp);
      sp -= 32u;
      continue;
    }
    if (sp >= 32u) break;
    const uint32_t nspill = W.nspill;
    if (nspill != 0u) {
      const uint32_t n = min(nspill, 32u);
      if (lane < n) {
        uint4 e = __ldcg(walk_region(S.w, round) + nspill - n + lane);
        e.w += shared_address(W.window);
        stack_put(W, sp + lane, e);
      }
      __syncwarp();
      if (lane == 0u) W.nspill = nspill - n;
      sp += n;
      continue;
    }
    if (W.more && !W.blocked) {
      if (W.cpos < W.cend)
        walk_roots<Batched>(S, W, lane, lt, sp, np);
      else if (W.lpos < W.lend)
        sp += walk_load<Batched>(round, sp);
      else
        walk_supply<Batched>(round);
      continue;
    }
    if (sp == 0u) {  // nothing left here (np == 0: settled above)
      walk_flush<Batched>(W.ncols);
      const bool more = W.more != 0u;
      __syncwarp();
      if (lane == 0u) {
        W.ncols = 0u;
        W.blocked = 0u;
      }
      if (!more) return kWalkDone;
      continue;
    }
    walk_step<Batched, false>(S.w.a.ks, S, W, lane, lt, sp, np);
    recent += 4u;  // few cells: look at the idle warps sooner
  }
  __syncwarp();
  if (lane == 0u) W.recent = recent;
  __syncwarp();
  return sp | (np << 16);
}

// The whole run: rounds separated by grid barriers (cooperative launch, every block resident),
// until a round hands nothing over.
template <bool Batched>
__global__ void __launch_bounds__(kWalkThreads, kWalkBlocksPerSm) k_walk(const __grid_constant__ WalkArgs w) {
  WalkSmem<Batched>& S = walk_shared<Batched>();
  WalkWarp<Batched>& W = walk_warp<Batched>();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u;
  for (uint32_t i = threadIdx.x; i < (uint32_t)kZigLayers; i += blockDim.x)
    S.zig[i] = make_uint2(__ldg(&w.a.zig->k[i]), __float_as_uint(__ldg(&w.a.zig->w[i])));
  for (uint32_t i = lane; i < kCols * kColWords; i += 32u) W.window[i] = 0u;
  for (uint32_t i = threadIdx.x; i < (uint32_t)(sizeof(WalkArgs) / 4u); i += blockDim.x)
    reinterpret_cast<uint32_t*>(&S.w)[i] = reinterpret_cast<const uint32_t*>(&w)[i];
  if (threadIdx.x == 0) S.finished = 0u;
  __syncthreads();
  for (uint32_t round = 0;; ++round) {
    // the control words two rounds on: last read in the round before this one
    if (blockIdx.x == 0 && threadIdx.x == 0) w.ctl->round[(round + 2u) & 3u] = WalkRound();
    if (lane == 0u) {
      W.cpos = W.cend = 0ull;
      W.lpos = W.lend = 0u;
      W.divisions = W.vanished = W.uncounted = 0ull;
      W.ncols = W.nspill = W.steps = W.polls = W.max_gen = W.blocked = W.taken = 0u;
      W.recent = kPollSteps - kFirstPoll;
      W.more = 1u;
    }
    __syncwarp();
    uint32_t sp = 0, np = 0, steps = 0;
    for (;;) {
      const uint32_t r = walk_manage<Batched>(round, sp, np, steps);
      if (r == kWalkDone) break;
      sp = r & 0xFFFFu;
      np = r >> 16;
      uint32_t left = kPollSteps;
#pragma unroll 1
      do {
        if (walk_step<Batched, true>(w.a.ks, S, W, lane, lt, sp, np) && np >= 32u) left = 1u;
      } while (--left != 0u && sp - 32u <= kStackRoom<Batched> - 32u);
      steps = kPollSteps - left;
    }
    __syncwarp();
    if (lane == 0u) {
      if (W.divisions) atomicAdd(&w.ctl->divisions, W.divisions);
      if (W.vanished) atomicAdd(&w.ctl->vanished, W.vanished);
      if (W.uncounted) atomicAdd(&w.ctl->uncounted, W.uncounted);
      if (W.max_gen) atomicMax(&w.ctl->max_gen, W.max_gen);
      // idle warps are reported by the eight
      if ((atomicAdd(&S.finished, 1u) & 7u) == 7u) atomicAdd(&w.ctl->round[round & 3u].idle, 8u);
    }
    if (!grid_barrier(&w.ctl->barrier[0], w.timeout_ns, w.a.error)) return;
    if (__ldcg(&w.ctl->round[round & 3u].handed) == 0ull) {  // a range is only given back together with cells
      if (blockIdx.x == 0 && threadIdx.x == 0) w.ctl->rounds = round + 1u;
      return;
    }
  }
}

}  // namespace
}  // namespace pc
