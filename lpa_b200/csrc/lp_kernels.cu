// Label-propagation kernels for sm_100a.
//
// One synchronous iteration reads lab_in and writes lab_out (double-buffered)
// for every vertex of degree > 0.  The update rule: the most frequent
// neighbour label, the smallest label on ties; vertices with degree >=
// cms_thr (cms_thr != 0) use a depth-4, width-1024 count-min sketch with
// seeded cm_hash rows (include/cms.cuh:96-132) and take the argmax of the
// sketch estimate over their neighbour labels, smallest label on ties.
//
// k_iterate and k_light are persistent kernels, each fed by a device work queue:
//   * heavy items (hubs the two-pass kernels do not take), one per block,
//     largest first: 256-bit segments decode in parallel (one thread each), ids
//     are staged in shared memory, labels are gathered with many loads in
//     flight, then counted in a shared (or global) table or the sketch;
//   * light items of up to 32 consecutive positions, one per warp: the lanes
//     decode the batch's segments into the warp's staging area, the warp
//     gathers all labels at once, then counts, a lane per vertex of degree
//     <= 32, the others one after another.
// The two-pass kernels (k_decode_two_pass, k_count_two_pass) write every
// neighbour label to a scratch and count from there; k_packed and
// k_packed_loop take the tiny vertices, a lane each.
// Every loop is bounded by the bits it consumes; malformed input sets the
// error word instead of trapping.
#include <type_traits>

#include "lp_kernels.cuh"
#include "noalloc.cuh"

namespace lpa_dev {

namespace {

// Epoch ranges of the shared tables: warp tables use [1, kLightEpochs), the
// block table [kLightEpochs, 65536), so a slot left by one mode never matches
// the other.
constexpr uint32_t kLightEpochs = 32768;
constexpr uint32_t kHeavyEpochFirst = 32768;

__device__ __forceinline__ uint32_t next_pow2(uint32_t x) { return x <= 1 ? 1u : (1u << (32 - __clz(x - 1))); }

struct Ctx {
  const uint32_t *lab_in;
  uint32_t *lab_out;
  unsigned long long *changed;
  uint32_t it;
  bool coherent;  // labels may change within the launch (batched graphs): read them through L2
};

// A label read: the non-coherent path when labels are fixed for the whole
// launch, else an L2 (ld.global.cg) read.
__device__ __forceinline__ uint32_t ld_label(const Ctx &c, uint32_t i) {
  return c.coherent ? __ldcg(c.lab_in + i) : __ldg(c.lab_in + i);
}

// An L2 cache policy that evicts the lines it is given last, and a load
// through L2 only (ld.global.cg) under such a policy.
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint32_t ld_cg_keep(const uint32_t *q, uint64_t pol) {
  uint32_t v;
  asm("ld.global.cg.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(q), "l"(pol));
  return v;
}

// A neighbour's label in a random gather: the lowest kHotIds ids (the hubs,
// in BFS order) through L1, every other id through L2 only, so that the
// scattered reads do not push the hot labels out of L1.
__device__ __forceinline__ uint32_t ld_label_gather(const Ctx &c, uint32_t i) {
  return (!c.coherent && i < kHotIds) ? __ldg(c.lab_in + i) : __ldcg(c.lab_in + i);
}

__device__ __forceinline__ Ctx resolve(const IterArgs &a) {
  Ctx c;
  c.it = iter_index(a);
  const uint32_t par = (a.parity0 + c.it) & 1u;
  c.lab_in = par ? a.labs1 : a.labs0;
  c.lab_out = par ? a.labs0 : a.labs1;
  c.changed = a.changed + (a.it_dev ? c.it : 0u);
  c.coherent = false;
  return c;
}

__device__ __forceinline__ void flush_changed(unsigned long long *counter, unsigned long long mine) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(counter, mine);
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, v, o);
    if (lane >= uint32_t(o)) v += t;
  }
  return v;
}

struct BlockSh {
  uint32_t pref[kThreads + 1];
  uint32_t left[kThreads];
  uint32_t wsum[kWarps];
  uint64_t red[kWarps];
  uint64_t ibase, rbase, last_end;
  uint32_t nseg_i, nseg_r, item, items, bad;
  uint32_t hepoch;  // epoch of the block's exact table
  uint32_t top;     // the global table's count of kTopLabel
};

// Block-wide exclusive scan of v into sh.pref; returns the total.
__device__ __forceinline__ uint32_t block_scan(BlockSh &sh, uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t incl = warp_incl_scan(v, lane);
  if (lane == 31) sh.wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kWarps ? sh.wsum[lane] : 0u;
    const uint32_t wi = warp_incl_scan(w, lane);
    if (lane < kWarps) sh.wsum[lane] = wi - w;
    if (lane == kWarps - 1) sh.pref[kThreads] = wi;
  }
  __syncthreads();
  sh.pref[threadIdx.x] = incl - v + sh.wsum[warp];
  __syncthreads();
  return sh.pref[kThreads];
}

// ------------------------------------------------------------ consumers ---
// A warp-uniform run of one label: a step whose real labels all equal the
// run's label only adds to the run's count (two ballots), so a vertex whose
// neighbours share one label touches its table once per label change, not
// once per step.  extend() is called by all 32 lanes.
struct WarpRun {
  uint32_t lab = kFull, cnt = 0;
  __device__ __forceinline__ bool extend(bool ok, uint32_t l) {
    const uint32_t okm = __ballot_sync(kFull, ok);
    if (__ballot_sync(kFull, ok && l == lab) != okm) return false;
    cnt += __popc(okm);
    return true;
  }
  // starts a new run at the label of the step's first real lane (the step
  // itself is counted by the caller)
  __device__ __forceinline__ void restart(bool ok, uint32_t l) {
    const uint32_t okm = __ballot_sync(kFull, ok);
    lab = __shfl_sync(kFull, l, __ffs(okm) - 1);
    cnt = 0;
  }
};

// Sinks are called warp-synchronously by every lane; ok marks a real label.
// The exact tables fold lanes holding the same label first (warp_merge), so a
// step whose lanes share a label touches the table once.
struct ExactSink {  // global table (key/count arrays, cleared after use)
  uint32_t *keys, *cnts, cap, *top;
  __device__ __forceinline__ void operator()(bool ok, uint32_t lab) const {
    const uint32_t w = warp_merge(ok, lab);
    if (w) table_add(keys, cnts, cap, top, lab, w);
  }
};

struct EpochSink {  // shared epoch table with a running argmax per thread
  EpochTable et;
  uint64_t *best;
  __device__ __forceinline__ void operator()(bool ok, uint32_t lab) const {
    const uint32_t w = warp_merge(ok, lab);
    if (w) {
      const uint64_t cand = pack_best(et.insert(lab, w), lab);
      if (cand > *best) *best = cand;
    }
  }
};

// Every lane adds its own label: the shared-memory atomics absorb the
// conflicts of lanes holding the same label for less than folding them first
// costs (fixed plan at R-MAT scale 24: 13.48 -> 13.02 ms per iteration).
struct CmsAddSink {
  uint32_t *cms;
  const uint32_t *seeds;
  uint32_t base;  // label_base of the vertex
  __device__ __forceinline__ void operator()(bool ok, uint32_t lab) const {
    if (ok) {
#pragma unroll
      for (int r = 0; r < kCmsDepth; r++)
        atomicAdd(&cms[r * kCmsWidth + (cm_hash(r, (lab - base) ^ seeds[r]) & (kCmsWidth - 1))], 1u);
    }
  }
};

// Second sketch pass: read-only, so every lane looks up its own label.
struct CmsBestSink {
  const uint32_t *cms;
  const uint32_t *seeds;
  uint32_t base;
  uint64_t *best;
  __device__ __forceinline__ void operator()(bool ok, uint32_t lab) const {
    if (ok) {
      // est <= the first row's counter: a label whose first counter cannot
      // beat this lane's best is not looked up further (fixed plan at R-MAT
      // scale 24: -0.1 ms per iteration)
      uint32_t est = cms[cm_hash(0, (lab - base) ^ seeds[0]) & (kCmsWidth - 1)];
      if (pack_best(est, lab) > *best) {
#pragma unroll
        for (int r = 1; r < kCmsDepth; r++) {
          const uint32_t v = cms[r * kCmsWidth + (cm_hash(r, (lab - base) ^ seeds[r]) & (kCmsWidth - 1))];
          est = v < est ? v : est;
        }
        const uint64_t cand = pack_best(est, lab);
        if (cand > *best) *best = cand;
      }
    }
  }
};

// Labels of the global ids src[0..total) into stage (src_labels: src holds
// the labels themselves).
__device__ __forceinline__ void block_gather_from(uint32_t *stage, const uint32_t *__restrict__ src, uint32_t total,
                                                  const Ctx &c, bool src_labels) {
  for (uint32_t k0 = threadIdx.x; k0 < total; k0 += 4 * kThreads) {
    uint32_t v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t k = k0 + u * kThreads;
      v[u] = k >= total ? 0u : (src_labels ? __ldcs(src + k) : ld_label_gather(c, __ldg(src + k)));
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t k = k0 + u * kThreads;
      if (k < total) stage[k] = v[u];
    }
  }
}

template <class Sink>
__device__ __forceinline__ void block_consume_stage(const uint32_t *stage, uint32_t total, const Sink &sink) {
  for (uint32_t k0 = 0; k0 < total; k0 += kThreads) {
    const uint32_t k = k0 + threadIdx.x;
    const bool ok = k < total;
    sink(ok, ok ? stage[k] : 0u);
  }
}

// Feeds every neighbour label of position p to sink, block-synchronously.
// Returns true when all labels ended up in stage[0..d) (one chunk, no
// intervals), so a second pass can read them from there.
template <class Sink>
__device__ bool heavy_produce(const IterArgs &a, const Ctx &c, BlockSh &sh, uint32_t *stage, uint32_t p,
                              uint32_t node, uint32_t d, bool from_scratch, const Sink &sink) {
  const DevGraph &g = a.g;
  const uint32_t t = threadIdx.x;
  if (p >= g.n_c || from_scratch) {
    // contiguous: the small CSR's ids, or the labels the two-pass pre-pass wrote
    const bool labels = p < g.n_c && a.scratch_labels;
    const uint32_t *src = labels ? a.scratch + a.arc_off[p] : g.small_nbr + g.small_off[p - g.n_c];
    for (uint32_t c0 = 0; c0 < d; c0 += kStage) {
      const uint32_t cnt = min(kStage, d - c0);
      block_gather_from(stage, src + c0, cnt, c, labels);
      __syncthreads();
      block_consume_stage(stage, cnt, sink);
      __syncthreads();
    }
    return false;
  }
  const uint64_t end = g.offsets[p + 1];
  bool bad = false;
  uint32_t my_items = 0;
  if (t == 0) {
    BitReader r;
    r.seek(g.words, g.offsets[p]);
    uint32_t ns = r.segcnt(bad);
    if (bad || r.pos() > end || ns > (end - r.pos()) / kSegBits + 1) {
      bad = true;
      ns = 0;
    }
    sh.nseg_i = ns;
    sh.ibase = r.pos();
    sh.last_end = r.pos();
    sh.bad = bad ? 1u : 0u;
    sh.items = 0;
  }
  __syncthreads();
  const uint32_t nseg_i = sh.nseg_i;
  const uint64_t ibase = sh.ibase;
  // ---- interval section: pairs decoded one per thread per step, flattened block-wide
  for (uint32_t j0 = 0; j0 < nseg_i; j0 += kThreads) {
    const uint32_t j = j0 + t;
    bool has = j < nseg_i;
    BitReader r;
    uint32_t cnt = 0, cc = 0, left = 0;
    const uint64_t q = ibase + uint64_t(kSegBits) * j;
    if (has) {
      if (q >= end) {
        bad = true;
        has = false;
      } else {
        r.seek(g.words, q);
        cnt = r.gamma(bad);
      }
    }
    while (__syncthreads_or(has && cc < cnt)) {
      uint32_t len = 0;
      if (has && cc < cnt) {
        const uint32_t l = r.gamma(bad);
        left = (cc == 0) ? zigzag_first(node, l) : left + l + 1u;
        len = r.gamma(bad) + kMinItv;
        cc++;
        if (bad || r.pos() > end || uint64_t(left) + len > g.n) {
          bad = true;
          len = 0;
          cnt = cc;
        }
      }
      sh.left[t] = left;
      const uint32_t total = block_scan(sh, len);
      if (len) left += len;
      for (uint32_t i0 = 0; i0 < total; i0 += 4 * kThreads) {
        uint32_t lab[4];
        bool ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t i = i0 + u * kThreads + t;
          ok[u] = i < total;
          lab[u] = 0;
          if (ok[u]) {
            uint32_t lo = 0, hi = kThreads - 1;
            while (lo < hi) {
              const uint32_t mid = (lo + hi + 1) >> 1;
              if (sh.pref[mid] <= i) lo = mid;
              else hi = mid - 1;
            }
            lab[u] = ld_label(c, sh.left[lo] + (i - sh.pref[lo]));
            my_items++;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) sink(ok[u], lab[u]);
      }
      __syncthreads();
    }
    if (has && j == nseg_i - 1) sh.last_end = r.pos();
  }
  __syncthreads();
  // ---- residual section: every warp walks its own 256-bit segments (lane per
  // segment, 32 per round) through its slice of the staging area; warps only
  // meet again at the end.
  if (t == 0) {
    BitReader r;
    r.seek(g.words, sh.last_end);
    uint32_t ns = r.segcnt(bad);
    if (bad || r.pos() > end || ns > (end - r.pos()) / kSegBits + 1) {
      bad = true;
      ns = 0;
    }
    sh.nseg_r = ns;
    sh.rbase = r.pos();
    sh.last_end = r.pos();
  }
  __syncthreads();
  const uint32_t nseg_r = sh.nseg_r;
  const uint64_t rbase = sh.rbase;
  const uint32_t lane = t & 31u, warp = t >> 5;
  uint32_t *wst = stage + warp * kWarpStage;
  bool single = true;  // this warp's labels all sit in its slice after one batch
  uint32_t staged = 0;
  int batches = 0;
  for (uint32_t j0 = warp * 32u; j0 < nseg_r; j0 += kWarps * 32u) {
    const uint32_t j = j0 + lane;
    bool has = j < nseg_r;
    BitReader r;
    uint32_t cnt = 0;
    if (has) {
      const uint64_t q = rbase + uint64_t(kSegBits) * j;
      if (q >= end) {
        bad = true;
        has = false;
      } else {
        r.seek(g.words, q);
        cnt = r.gamma(bad);
        if (bad || cnt > kWarpStage) {
          bad = true;
          cnt = 0;
        }
      }
    }
    uint32_t done = ~__ballot_sync(kFull, has);
    while (done != kFull) {
      const bool pending = !((done >> lane) & 1u);
      const uint32_t sc = pending ? cnt : 0u;
      const uint32_t incl = warp_incl_scan(sc, lane);
      const bool in_batch = pending && incl <= kWarpStage;
      const uint32_t batch = __ballot_sync(kFull, in_batch);
      const uint32_t total = __shfl_sync(kFull, incl, 31 - __clz(batch));
      if (in_batch) {
        // ids are clamped to n - 1, so every gather stays in range; a
        // segment's ids ascend, so its last one is its largest, and it and the
        // segment's end are tested once, after the last code (the stream was
        // validated code by code when the handle was created)
        const uint32_t nmax = uint32_t(g.n - 1);
        uint32_t o = incl - sc, v = 0;
        if (cnt) {
          v = zigzag_first(node, r.zeta3(bad));
          wst[o++] = min(v, nmax);
        }
        for (uint32_t cc = 1; cc < cnt; cc++) {
          v += r.zeta3(bad) + 1u;
          wst[o++] = min(v, nmax);
        }
        if (cnt && (v > nmax || r.pos() > end)) bad = true;
        my_items += cnt;
        if (j == nseg_r - 1) sh.last_end = r.pos();
      }
      __syncwarp();
      for (uint32_t k0 = lane; k0 < total; k0 += 256) {
        uint32_t lv[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t k = k0 + 32 * u;
          lv[u] = k < total ? ld_label_gather(c, wst[k]) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t k = k0 + 32 * u;
          if (k < total) wst[k] = lv[u];
        }
      }
      __syncwarp();
      for (uint32_t k0 = 0; k0 < total; k0 += 32) {
        const uint32_t k = k0 + lane;
        const bool ok = k < total;
        sink(ok, ok ? wst[k] : 0u);
      }
      __syncwarp();
      staged = total;
      batches++;
      done |= batch;
    }
  }
  if (batches > 1) single = false;
  if (my_items) atomicAdd(&sh.items, my_items);
  if (bad) sh.bad = 1;
  const bool all_single = __syncthreads_and(single) != 0;
  if (t == 0 && (sh.bad || sh.last_end != end || sh.items != d)) set_error(a.err, kErrBadStream);
  if (lane == 0) sh.wsum[warp] = staged;
  __syncthreads();
  return nseg_i == 0 && all_single;
}

// Second pass over labels left in the warps' slices by heavy_produce.
template <class Sink>
__device__ __forceinline__ void heavy_consume_staged(BlockSh &sh, const uint32_t *stage, const Sink &sink) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t *wst = stage + warp * kWarpStage;
  const uint32_t total = sh.wsum[warp];
  for (uint32_t k0 = 0; k0 < total; k0 += 32) {
    const uint32_t k = k0 + lane;
    const bool ok = k < total;
    sink(ok, ok ? wst[k] : 0u);
  }
}

// One heavy vertex by the whole block.
__device__ void heavy_vertex(const IterArgs &a, const Ctx &c, BlockSh &sh, uint32_t *stage, uint32_t *tab,
                             uint32_t seg, uint32_t p, bool from_scratch, unsigned long long &changed) {
  const DevGraph &g = a.g;
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint32_t node = g.vertices[p];
  const uint32_t d = g.deg[p];
  const uint32_t old = ld_label(c, node);
  if (a.cursor && from_scratch && p < g.n_c && t == 0) a.cursor[p] = 0u;  // the pre-pass's output cursor, for the next iteration
  if (d == 0) return;
  uint64_t best = 0;
  if (a.cms_thr != 0 && d >= a.cms_thr) {
    // the sketch shares its memory with the exact tables, whose slots are
    // never cleared: zero the counters first
    uint32_t *cms = tab;
    for (uint32_t i = t; i < kCmsDepth * kCmsWidth; i += kThreads) cms[i] = 0u;
    __syncthreads();
    const uint32_t lb = label_base(a, node);
    const bool staged = heavy_produce(a, c, sh, stage, p, node, d, from_scratch, CmsAddSink{cms, a.seeds, lb});
    __syncthreads();
    CmsBestSink s2{cms, a.seeds, lb, &best};
    if (staged) heavy_consume_staged(sh, stage, s2);
    else if ((p >= g.n_c || from_scratch) && d <= kStage) block_consume_stage(stage, d, s2);
    else heavy_produce(a, c, sh, stage, p, node, d, from_scratch, s2);
    __syncthreads();
    // leave no counter behind that an epoch table could read as its own slot
    for (uint32_t i = t; i < kCmsDepth * kCmsWidth; i += kThreads) cms[i] = 0u;
  } else if (d <= kBlockMaxSmemDeg) {
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(tab);
    if (t == 0) {
      if (++sh.hepoch >= 65536u) sh.hepoch = 0;
    }
    __syncthreads();
    if (sh.hepoch == 0) {  // epochs used up: start the block table over
      for (uint32_t i = t; i < kTableSlots; i += kThreads) slots[i] = 0ull;
      __syncthreads();
      if (t == 0) sh.hepoch = kHeavyEpochFirst;
      __syncthreads();
    }
    const EpochTable et{slots, next_pow2(2 * d), sh.hepoch};
    heavy_produce(a, c, sh, stage, p, node, d, from_scratch, EpochSink{et, &best});
    __syncthreads();
  } else {
    const uint32_t cap = next_pow2(2 * d);
    if (a.gtab_slots == 0 || cap > a.gtab_slots) {
      if (t == 0) set_error(a.err, kErrCapacity);
      return;
    }
    uint32_t *keys = a.gtab + uint64_t(blockIdx.x) * 2 * a.gtab_slots;
    uint32_t *cnts = keys + a.gtab_slots;
    if (t == 0) sh.top = 0;
    __syncthreads();
    heavy_produce(a, c, sh, stage, p, node, d, from_scratch, ExactSink{keys, cnts, cap, &sh.top});
    __syncthreads();
    if (t == 0 && sh.top) best = pack_best(sh.top, kTopLabel);
    for (uint32_t i = t; i < cap; i += kThreads) {
      const uint32_t kk = keys[i];
      if (kk) {
        const uint64_t cand = pack_best(cnts[i], kk - 1u);
        best = cand > best ? cand : best;
        keys[i] = 0u;
        cnts[i] = 0u;
      }
    }
  }
  best = warp_max_u64(best);
  if (lane == 0) sh.red[warp] = best;
  __syncthreads();
  if (t == 0) {
    uint64_t b = 0;
    for (int w = 0; w < kWarps; w++) b = sh.red[w] > b ? sh.red[w] : b;
    const uint32_t nl = b ? best_label(b) : old;
    c.lab_out[node] = nl;
    changed += (nl != old);
    if (a.seg_changed && nl != old) atomicAdd(a.seg_changed + seg, 1u);
  }
  __syncthreads();
}

// Decodes the compressed vertices of a warp batch into stage (ids).  Lane l
// owns the batch vertex in lane l: it reads that vertex's section headers and
// writes its interval items (lane per vertex); then the batch's residual
// segments are spread over the lanes (lane per 256-bit segment, 32 per
// round) and placed with warp prefix sums over the segments' item counts.
// Returns false (after filling every region with in-range ids) on a
// malformed stream.
__device__ bool warp_decode_batch(const DevGraph &g, uint32_t *stage, bool active, uint32_t p, uint32_t node,
                                  uint32_t d, uint32_t base, uint32_t lane) {  // stage: shared or global
  bool bad = false;
  uint32_t nres = 0, itv = 0;
  uint64_t rbase = 0, end = 0;
  if (active && d) {
    end = g.offsets[p + 1];
    BitReader r;
    r.seek(g.words, g.offsets[p]);
    uint32_t ns = r.segcnt(bad);
    const uint64_t ib = r.pos();
    uint64_t last = r.pos();
    if (bad || r.pos() > end || ns > (end - r.pos()) / kSegBits + 1) {
      bad = true;
      ns = 0;
    }
    for (uint32_t j = 0; j < ns && !bad; j++) {
      const uint64_t q = ib + uint64_t(kSegBits) * j;
      if (q >= end) {
        bad = true;
        break;
      }
      if (j) r.seek(g.words, q);
      const uint32_t cnt = r.gamma(bad);
      uint32_t left = 0;
      for (uint32_t c = 0; c < cnt && !bad; c++) {
        const uint32_t l = r.gamma(bad);
        left = (c == 0) ? zigzag_first(node, l) : left + l + 1u;
        const uint32_t len = r.gamma(bad) + kMinItv;
        if (bad || r.pos() > end || uint64_t(left) + len > g.n || uint64_t(itv) + len > d) {
          bad = true;
          break;
        }
        for (uint32_t k = 0; k < len; k++) stage[base + itv + k] = left + k;
        itv += len;
        left += len;
      }
      last = r.pos();
    }
    if (ns) r.seek(g.words, last);
    if (!bad) {
      nres = r.segcnt(bad);
      rbase = r.pos();
      if (bad || r.pos() > end || nres > (end - r.pos()) / kSegBits + 1) {
        bad = true;
        nres = 0;
      } else if (nres == 0 && r.pos() != end) {
        bad = true;
      }
    }
  }
  const uint32_t seg_incl = warp_incl_scan(nres, lane);
  const uint32_t seg_excl = seg_incl - nres;
  const uint32_t S = __shfl_sync(kFull, seg_incl, 31);
  uint32_t res_done = 0;
  for (uint32_t r0 = 0; r0 < S; r0 += 32) {
    const uint32_t f = r0 + lane;
    const bool has = f < S;
    // owner: the last lane whose first segment is <= f
    uint32_t lo = 0, hi = 31;
#pragma unroll
    for (int step = 0; step < 5; step++) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      const uint32_t e = __shfl_sync(kFull, seg_excl, mid);
      if (e <= f) lo = mid;
      else hi = mid - 1;
    }
    const uint32_t o = lo;
    const uint32_t eo = __shfl_sync(kFull, seg_excl, o);
    const uint32_t no = __shfl_sync(kFull, nres, o);
    const uint64_t rb = __shfl_sync(kFull, rbase, o);
    const uint64_t en = __shfl_sync(kFull, end, o);
    const uint32_t ndo = __shfl_sync(kFull, node, o);
    const uint32_t bo = __shfl_sync(kFull, base, o);
    const uint32_t io = __shfl_sync(kFull, itv, o);
    const uint32_t dd = __shfl_sync(kFull, d, o);
    const uint32_t rdo = __shfl_sync(kFull, res_done, o);
    const uint32_t j = f - eo;
    BitReader rr;
    uint32_t cnt = 0;
    if (has) {
      const uint64_t q = rb + uint64_t(kSegBits) * j;
      if (q >= en) {
        bad = true;
      } else {
        rr.seek(g.words, q);
        cnt = rr.gamma(bad);
        if (bad || cnt > dd) {
          bad = true;
          cnt = 0;
        }
      }
    }
    const uint32_t c_incl = warp_incl_scan(cnt, lane);
    const uint32_t c_excl = c_incl - cnt;
    const uint32_t fo = (eo > r0 ? eo : r0) - r0;  // the owner's first lane in this round
    const uint32_t at_fo = __shfl_sync(kFull, c_excl, fo);
    if (has && !bad) {
      const uint32_t rel = io + rdo + (c_excl - at_fo);  // item offset inside the owner's region
      if (uint64_t(rel) + cnt > dd) {
        bad = true;
      } else {
        // clamped ids, one range and end test per segment (as heavy_produce)
        const uint32_t nmax = uint32_t(g.n - 1);
        uint32_t v = 0;
        if (cnt) {
          v = zigzag_first(ndo, rr.zeta3(bad));
          stage[bo + rel] = min(v, nmax);
        }
        for (uint32_t c = 1; c < cnt; c++) {
          v += rr.zeta3(bad) + 1u;
          stage[bo + rel + c] = min(v, nmax);
        }
        if (cnt && (v > nmax || rr.pos() > en)) bad = true;
      }
      if (j == no - 1 && rr.pos() != en) bad = true;
    }
    // owners advance by the items of their segments in this round
    const uint32_t fv = (seg_excl > r0 ? seg_excl : r0) - r0;
    const uint32_t lv_end = (seg_incl < r0 + 32 ? seg_incl : r0 + 32);
    const bool mine = nres && seg_incl > r0 && seg_excl < r0 + 32;
    const uint32_t lv = mine ? lv_end - r0 - 1 : 0u;
    const uint32_t a1 = __shfl_sync(kFull, c_incl, lv);
    const uint32_t a0 = __shfl_sync(kFull, c_excl, mine ? fv : 0u);
    if (mine) res_done += a1 - a0;
  }
  if (active && d && itv + res_done != d) bad = true;
  if (__any_sync(kFull, bad)) {
    if (active)
      for (uint32_t k = 0; k < d; k++) stage[base + k] = node;
    __syncwarp();
    return false;
  }
  return true;
}

// Up to 32 consecutive positions [p0, p1) by one warp.
// kSlots: the slots of the warp's table.
template <uint32_t kSlots>
__device__ void light_chunk(const IterArgs &a, const Ctx &c, uint32_t *stage, unsigned long long *slots,
                            uint32_t &epoch, uint32_t seg, uint32_t p0, uint32_t p1, int variant,
                            unsigned long long &changed) {
  const DevGraph &g = a.g;
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t cap_stage = kWarpStage;
  const uint32_t p = p0 + lane;
  const bool valid = p < p1;
  const uint32_t node = valid ? g.vertices[p] : 0u;
  uint32_t d = valid ? g.deg[p] : 0u;
  const uint32_t old = valid ? ld_label(c, node) : 0u;
  const bool cgr = p0 < g.n_c;  // chunks never straddle the compressed / small boundary
  const bool decode = cgr && variant != kVarTwoPass;
  if (a.cursor && cgr && !decode && valid) a.cursor[p] = 0u;  // the pre-pass's output cursor, for the next iteration
  if (d > cap_stage || (variant == kVarPacked && d > kV2MaxDeg) || d > kV1MaxDeg) {
    set_error(a.err, kErrCapacity);
    d = 0;
  }
  // contiguous id source of the chunk when it is not decoded here
  const uint32_t *src = nullptr;
  if (!decode) src = cgr ? a.scratch + a.arc_off[p0] : g.small_nbr + g.small_off[p0 - g.n_c];
  uint32_t src_skip = 0;  // ids consumed by earlier batches of this chunk
  uint32_t done = ~__ballot_sync(kFull, valid);
  uint32_t my_changed = 0;
  while (done != kFull) {
    const bool pending = !((done >> lane) & 1u);
    const uint32_t sd = pending ? d : 0u;
    const uint32_t incl = warp_incl_scan(sd, lane);
    const bool in_batch = pending && incl <= cap_stage;
    const uint32_t batch = __ballot_sync(kFull, in_batch);
    const uint32_t hi = 32 - __clz(batch);
    const uint32_t total = __shfl_sync(kFull, incl, hi - 1);
    const uint32_t base = incl - sd;
    // 1. ids: the batch decoded by all lanes together
    if (decode && !warp_decode_batch(g, stage, in_batch, p, node, d, base, lane) && lane == 0)
      set_error(a.err, kErrBadStream);
    __syncwarp();
    // 2. labels: every load of the batch in flight together
    for (uint32_t k0 = lane; k0 < total; k0 += 256) {
      uint32_t v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint32_t k = k0 + 32 * u;
        v[u] = k >= total ? 0u
                          : (decode ? ld_label_gather(c, stage[k])
                                    : (cgr && a.scratch_labels ? __ldcs(src + src_skip + k)
                                                               : ld_label_gather(c, __ldg(src + src_skip + k))));
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint32_t k = k0 + 32 * u;
        if (k < total) stage[k] = v[u];
      }
    }
    __syncwarp();
    // 3. count
    // vertices of degree <= 32: a lane each; one whose labels all agree takes
    // that label at once
    uint32_t nl = old;
    const bool few = in_batch && d <= 32;
    bool mixed = false;
    if (few && d) {
      nl = stage[base];
      for (uint32_t j = 1; j < d; j++) mixed |= stage[base + j] != nl;
    }
    if (uint32_t rest = __ballot_sync(kFull, mixed)) {
      if (one_by_one(__popc(rest), __reduce_max_sync(kFull, mixed ? d : 0u))) {
        for (; rest; rest &= rest - 1u) {
          const uint32_t l = uint32_t(__ffs(rest) - 1);
          const uint32_t x = warp_mode(stage + __shfl_sync(kFull, base, l), __shfl_sync(kFull, d, l));
          if (lane == l) nl = x;
        }
      } else if (mixed) {
        nl = lane_mode(stage + base, d);
      }
    }
    if (few) {
      c.lab_out[node] = nl;
      my_changed += (nl != old);
    }
    // the others by the warp, one after another
    for (uint32_t m = __ballot_sync(kFull, in_batch && d > 32); m; m &= m - 1u) {
      const uint32_t j = __ffs(m) - 1;
      const uint32_t dv = __shfl_sync(kFull, d, j);
      const uint32_t bv = __shfl_sync(kFull, base, j);
      const uint32_t nodev = __shfl_sync(kFull, node, j);
      const uint32_t oldv = __shfl_sync(kFull, old, j);
      // epoch table: no clearing, running argmax from the returned counts.  A
      // vertex with more labels than slots is counted in 2, 4, ... parts told
      // apart by the top bits of the slot hash.
      uint64_t bp = 0;
      for (uint32_t lg = dv <= kSlots ? 0u : dv <= 2 * kSlots - kSlots / 4 ? 1u : 2u;; lg += 2) {
        bool full = false;
        bp = 0;
        for (uint32_t part = 0; part < 1u << lg && !full; part++) {
          if (++epoch >= kLightEpochs) {
            for (uint32_t i = lane; i < kSlots; i += 32) slots[i] = 0ull;
            __syncwarp();
            epoch = 1;
          }
          const EpochTable et{slots, min(next_pow2(2 * dv), kSlots), epoch};
          const auto ins = [&](uint32_t lab, uint32_t w) {
            const uint32_t n = et.insert(lab, w);
            full |= n == 0u;
            const uint64_t cand = pack_best(n, lab);
            bp = cand > bp ? cand : bp;
          };
          // a step of one label extends the current run (fixed plan at R-MAT
          // scale 24: 13.48 -> 13.21 ms per iteration)
          WarpRun run;
          for (uint32_t k0 = 0; k0 < dv; k0 += 32) {
            const uint32_t k = k0 + lane;
            bool ok = k < dv;
            const uint32_t lab = ok ? stage[bv + k] : kFull;
            if (lg) ok = ok && slot_hash(lab) >> (32u - lg) == part;
            if (run.extend(ok, lab)) continue;
            if (run.cnt && lane == 0) ins(run.lab, run.cnt);
            run.restart(ok, lab);
            const uint32_t w = warp_merge(ok, lab);
            if (w) ins(lab, w);
          }
          if (run.cnt && lane == 0) ins(run.lab, run.cnt);
          full = __any_sync(kFull, full);
        }
        if (!full) break;
      }
      const uint32_t bestl = best_label(warp_max_u64(bp));
      __syncwarp();
      if (lane == 0) {
        c.lab_out[nodev] = bestl;
        my_changed += (bestl != oldv);
      }
    }
    __syncwarp();
    src_skip += total;
    done |= batch;
  }
  changed += my_changed;
  if (a.seg_changed) {
    const uint32_t s = __reduce_add_sync(kFull, my_changed);
    if (lane == 0 && s) atomicAdd(a.seg_changed + seg, s);
  }
}

// The block variant over one plan segment.  A vertex that one warp's table
// and staging area hold (exact, degree <= kV1MaxDeg) is decoded and counted
// by one warp, eight of them side by side: its 256-bit segments number at
// most 64, so one vertex per block would leave most of the block idle while
// a few lanes decode.  A hub (larger, or at the sketch threshold) takes the
// whole block, whose 256 threads then decode its segments in parallel.
__device__ void block_segment(const IterArgs &a, const Ctx &c, BlockSh &sh, uint32_t *stage, uint32_t *tab,
                              uint32_t *wstage, unsigned long long *wslots, uint32_t &wepoch, uint32_t s,
                              const Seg sg, bool from_scratch, unsigned long long &changed) {
  const DevGraph &g = a.g;
  const uint32_t t = threadIdx.x, warp = t >> 5;
  bool fits = true;
  for (uint32_t p = sg.begin + t; p < sg.end; p += kThreads) {
    const uint32_t d = g.deg[p];
    fits &= d <= kV1MaxDeg && !(a.cms_thr != 0 && d >= a.cms_thr);
  }
  if (__syncthreads_and(fits)) {
    const int v = from_scratch ? kVarTwoPass : kVarWarp;
    for (uint32_t p = sg.begin + warp; p < sg.end; p += kWarps) light_chunk<kWarpSlots>(a, c, wstage, wslots, wepoch, s, p, p + 1, v, changed);
    __syncthreads();  // the block's shared memory is free for the next item
    return;
  }
  for (uint32_t p = sg.begin; p < sg.end; p++) heavy_vertex(a, c, sh, stage, tab, s, p, from_scratch, changed);
}

}  // namespace

// Widens the kernel's busy span in a.ktime by this warp's start or end.
__device__ __forceinline__ void busy_mark(const IterArgs &a, int kernel, bool end) {
  if (a.ktime && (threadIdx.x & 31u) == 0) {
    const unsigned long long t = global_ns();
    if (end) atomicMax(a.ktime + kBusyKernels + kernel, t);
    else atomicMin(a.ktime + kernel, t);
  }
}

__global__ void __launch_bounds__(kThreads, 2) k_iterate(IterArgs a) {
  extern __shared__ uint32_t smem[];
  __shared__ BlockSh sh;
  uint32_t *stage = smem;         // kStage words
  uint32_t *tab = smem + kStage;  // kTableSlots keys + kTableSlots counts (or the sketch)
  const uint32_t t = threadIdx.x, warp = t >> 5;
  for (uint32_t i = t; i < 2 * kTableSlots; i += kThreads) tab[i] = 0u;
  if (t == 0) sh.hepoch = kHeavyEpochFirst;
  __syncthreads();
  const Ctx c = resolve(a);
  busy_mark(a, 2, false);
  unsigned long long changed = 0;
  uint32_t *qctr = a.work + kWorkCounters * (a.it_dev ? c.it : 0u) + kWqHeavy;

  // per-warp staging and exact table of the warp-scope paths
  unsigned long long *wslots = reinterpret_cast<unsigned long long *>(tab) + warp * kWarpSlots;
  uint32_t *wstage = stage + warp * kWarpStage;
  uint32_t wepoch = 0;

  // heavy items: one segment per block (largest first).  The next item is
  // claimed before the current one runs and its bits are prefetched into L2.
  if (t == 0) {
    const uint32_t i0 = atomicAdd(qctr, 1u);
    sh.item = i0;
    if (i0 < a.n_heavy) prefetch_l2(reinterpret_cast<const void *>(a.heavy[i0].pf_addr), a.heavy[i0].pf_bytes);
  }
  __syncthreads();
  uint32_t next = sh.item;
  for (;;) {
    const uint32_t i = next;
    __syncthreads();
    if (i >= a.n_heavy) break;
    if (t == 0) {
      const uint32_t in = atomicAdd(qctr, 1u);
      sh.item = in;
      if (in < a.n_heavy) prefetch_l2(reinterpret_cast<const void *>(a.heavy[in].pf_addr), a.heavy[in].pf_bytes);
    }
    __syncthreads();
    next = sh.item;
    const uint32_t s = a.heavy[i].seg;
    const bool from_scratch = a.seg_var[s] == kVarTwoPass;
    const Seg sg = a.segs[s];
    const long long t0 = clock64();
    block_segment(a, c, sh, stage, tab, wstage, wslots, wepoch, s, sg, from_scratch, changed);
    if (a.seg_cycles && t == 0)
      atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + s),
                (unsigned long long)((clock64() - t0) * kWarps * a.cw_iterate));
  }

  busy_mark(a, 2, true);
  flush_changed(c.changed, changed);
}

// The light items of the warp, packed and block variants, a warp each.  A
// kernel of its own, apart from the heavy items' registers and 12 KB of
// shared memory per warp: 8 KB here (1024 staged labels, 512 table slots) and
// three blocks per SM instead of two (light items of the fixed plan: R-MAT scale
// 20 264 -> 208 us, 22 1135 -> 891 us, 4M-vertex copy model 950 -> 624 us).
__global__ void __launch_bounds__(kThreads, 3) k_light(IterArgs a) {
  extern __shared__ __align__(16) unsigned long long lsmem[];
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  unsigned long long *wslots = lsmem + warp * kLightSlots;
  uint32_t *wstage = reinterpret_cast<uint32_t *>(lsmem + kWarps * kLightSlots) + warp * kWarpStage;
  for (uint32_t i = lane; i < kLightSlots; i += 32) wslots[i] = 0ull;
  __syncwarp();
  const Ctx c = resolve(a);
  busy_mark(a, 2, false);
  unsigned long long changed = 0;
  uint32_t *qctr = a.work + kWorkCounters * (a.it_dev ? c.it : 0u) + kWqLight;
  uint32_t wepoch = 0;
  // light items, one at a time: a warp's first is its own, the others come
  // from the queue.  It knows its next item while it runs one (claimed a round
  // earlier, its range prefetched into L2).
  const uint32_t own = gridDim.x * kWarps;
  const auto claim = [&]() {
    uint32_t x = 0;
    if (lane == 0) x = atomicAdd(qctr, 1u);
    return own + __shfl_sync(kFull, x, 0);
  };
  WorkItem wi{};
  uint32_t cur = warp * gridDim.x + blockIdx.x, ahead = a.n_light > own ? claim() : a.n_light;
  if (cur < a.n_light) wi = a.light[cur];
  while (cur < a.n_light) {
    WorkItem wn{};
    if (ahead < a.n_light) {
      wn = a.light[ahead];
      if (lane == 0) prefetch_l2(reinterpret_cast<const void *>(wn.pf_addr), wn.pf_bytes);
    }
    uint32_t x = 0;  // the claim after that; not waited for until the item is done
    if (lane == 0 && ahead < a.n_light) x = atomicAdd(qctr, 1u);
    const long long t0 = clock64();
    light_chunk<kLightSlots>(a, c, wstage, wslots, wepoch, wi.seg, wi.p0, wi.p0 + wi.np, a.seg_var[wi.seg], changed);
    if (a.seg_cycles && lane == 0)
      atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + wi.seg),
                (unsigned long long)((clock64() - t0) * a.cw_light));
    cur = ahead;
    wi = wn;
    ahead = ahead < a.n_light ? own + __shfl_sync(kFull, x, 0) : ahead;
  }
  busy_mark(a, 2, true);
  flush_changed(c.changed, changed);
}

cudaError_t prepare_light(int *blocks) {
  cudaError_t e = cudaFuncSetAttribute(k_light, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kLightSmemBytes));
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_light, kThreads, kLightSmemBytes);
  return e;
}

enum LabelLoad : int { kLdShared, kLdFenced };  // packed_vertex
template <int kLoad>
__device__ __forceinline__ uint32_t packed_vertex(const IterArgs &a, const Ctx &c, uint32_t p, uint32_t *lab);

// Many graphs, one persistent launch.  A ring queue holds (graph,
// iteration, segment) items; iteration 0 of every graph is queued by the
// host.  The block that finishes the last item of a graph's iteration reads
// that iteration's changed count and either retires the graph or queues all
// its segments for the next iteration, so an item never waits on another
// item.  Blocks wait (bounded) only on an empty queue slot.  Labels change
// during the launch, so they are read through L2.
__global__ void __launch_bounds__(kThreads, 2) k_batch(BatchArgs b) {
  extern __shared__ uint32_t smem[];
  __shared__ BlockSh sh;
  __shared__ IterArgs ia;
  __shared__ unsigned long long s_item, s_enq_base;
  __shared__ uint32_t s_last, s_enq;
  uint32_t *stage = smem;
  uint32_t *tab = smem + kStage;
  const uint32_t t = threadIdx.x, warp = t >> 5;
  for (uint32_t i = t; i < 2 * kTableSlots; i += kThreads) tab[i] = 0u;
  if (t == 0) sh.hepoch = kHeavyEpochFirst;
  __syncthreads();
  unsigned long long *wslots = reinterpret_cast<unsigned long long *>(tab) + warp * kWarpSlots;
  uint32_t *wstage = stage + warp * kWarpStage;
  uint32_t wepoch = 0;
  for (;;) {
    if (t == 0) {
      const unsigned long long idx = atomicAdd(b.head, 1ull);
      volatile unsigned long long *slot = b.queue + (idx % b.cap);
      unsigned long long e = *slot;
      unsigned long long spins = 0;
      while (e == kQueueEmpty) {
        if (*reinterpret_cast<volatile uint32_t *>(b.active) == 0u) break;
        if (++spins > b.spin_limit) {
          set_error(b.err, kErrTimeout);
          break;
        }
        __nanosleep(200);
        e = *slot;
      }
      if (e != kQueueEmpty) *slot = kQueueEmpty;
      __threadfence();
      s_item = e;
    }
    __syncthreads();
    const unsigned long long e = s_item;
    if (e == kQueueEmpty) break;
    const uint32_t gi = uint32_t(e >> 44), it = uint32_t(e >> 32) & 0xFFFu, s = uint32_t(e);
    if (t == 0) {
      const BatchGraph &bg = b.graphs[gi];
      ia = IterArgs{};  // every field this launch does not use is zero (null): no scratch
      ia.g = bg.g;
      ia.labs0 = bg.labs0;
      ia.labs1 = bg.labs1;
      ia.parity0 = 0;
      ia.it_dev = nullptr;
      ia.changed = b.changed + gi;
      ia.work = nullptr;
      ia.err = b.err;
      ia.segs = bg.segs;
      ia.seg_var = bg.seg_var;
      ia.seg_cycles = nullptr;
      ia.seg_changed = nullptr;
      ia.cms_thr = b.cms_thr;
      for (int r = 0; r < kCmsDepth; r++) ia.seeds[r] = b.seeds[r];
      ia.scratch = nullptr;
      ia.arc_off = nullptr;
      ia.scratch_labels = 0;
      ia.groups = nullptr;
      ia.n_groups = 0;
      ia.pidx = nullptr;
      ia.cursor = nullptr;
      ia.ktime = nullptr;
      ia.packed = nullptr;
      ia.n_packed = 0;
      ia.gtab = b.gtab;
      ia.gtab_slots = b.gtab_slots;
      ia.gbase = nullptr;  // every graph has its own labels
      ia.n_gbase = 0;
    }
    __syncthreads();
    Ctx c;
    c.it = it;
    c.lab_in = (it & 1u) ? ia.labs1 : ia.labs0;
    c.lab_out = (it & 1u) ? ia.labs0 : ia.labs1;
    c.changed = ia.changed;
    c.coherent = true;
    unsigned long long changed = 0;
    const Seg sg = ia.segs[s];
    const int v = ia.seg_var[s];
    if (v == kVarBlock || v == kVarTwoPass) {
      block_segment(ia, c, sh, stage, tab, wstage, wslots, wepoch, s, sg, false, changed);
    } else if (v == kVarPackedLanes) {
      // a tiny segment: one thread per position (<= 256 positions)
      if (sg.begin + t < sg.end) changed += packed_vertex<kLdShared>(ia, c, sg.begin + t, stage + t * kPackedMaxDeg);
    } else {
      // light segments hold at most 256 positions: the same share for every warp
      const uint32_t per = (sg.end - sg.begin + kWarps - 1) / kWarps, p0 = sg.begin + warp * per;
      if (p0 < sg.end) light_chunk<kWarpSlots>(ia, c, wstage, wslots, wepoch, s, p0, min(sg.end, p0 + per), v, changed);
    }
    flush_changed(c.changed, changed);
    __threadfence();
    __syncthreads();
    if (t == 0) {
      const uint32_t nseg = b.graphs[gi].nseg;
      s_last = (atomicAdd(b.done_items + gi, 1u) + 1u == nseg) ? 1u : 0u;
      s_enq = 0;
      if (s_last) {
        __threadfence();
        const unsigned long long ch = atomicExch(b.changed + gi, 0ull);
        b.done_items[gi] = 0;
        b.iters[gi] = it + 1;
        const bool stop = (b.early_exit && ch == 0ull) || it + 1 >= b.max_iter;
        if (stop) {
          __threadfence();
          atomicSub(b.active, 1u);
        } else {
          s_enq_base = atomicAdd(b.tail, (unsigned long long)nseg);
          s_enq = nseg;
        }
      }
    }
    __syncthreads();
    if (s_enq) {
      const unsigned long long tag = (uint64_t(gi) << 44) | (uint64_t(it + 1) << 32);
      for (uint32_t k = t; k < s_enq; k += kThreads) {
        __threadfence();
        b.queue[(s_enq_base + k) % b.cap] = tag | k;
      }
    }
    __syncthreads();
  }
}

__global__ void k_batch_init(const BatchGraph *graphs, uint32_t ngraphs) {
  for (uint32_t gi = blockIdx.x; gi < ngraphs; gi += gridDim.x) {
    const BatchGraph &bg = graphs[gi];
    for (uint64_t v = threadIdx.x; v < bg.g.n; v += blockDim.x) {
      bg.labs0[v] = uint32_t(v);
      bg.labs1[v] = uint32_t(v);
    }
  }
}

// The d ids of a vertex of degree d <= kPackedRegs with the commonest layout
// (no intervals, one residual segment, at most 128 bits, gaps below 2^24), in
// registers: the count is known, so the headers are compared, not decoded, and
// the codes come from a 128-bit window without refills or position arithmetic.
// False when the vertex is not of that layout (the walk takes it).
constexpr uint32_t kPackedRegs = 8;
__device__ __forceinline__ bool packed_ids(const DevGraph &g, uint32_t p, uint32_t node, uint32_t d,
                                           uint32_t (&id)[kPackedRegs]) {
  const uint64_t o0 = g.offsets[p], len = g.offsets[p + 1] - o0;
  if (len > 128) return false;
  const uint32_t *w = g.words + (o0 >> 5);
  const uint32_t s = uint32_t(o0) & 31u, bits = s + uint32_t(len);
  // words past the vertex's last are never needed
  const uint32_t w0 = __ldg(w), w1 = bits > 32 ? __ldg(w + 1) : 0u, w2 = bits > 64 ? __ldg(w + 2) : 0u,
                 w3 = bits > 96 ? __ldg(w + 3) : 0u, w4 = bits > 128 ? __ldg(w + 4) : 0u;
  uint32_t x0 = __funnelshift_l(w1, w0, s), x1 = __funnelshift_l(w2, w1, s), x2 = __funnelshift_l(w3, w2, s),
           x3 = __funnelshift_l(w4, w3, s);
  uint32_t used = 0;
  const auto skip = [&](uint32_t k) {  // k <= 32
    x0 = __funnelshift_lc(x1, x0, k);
    x1 = __funnelshift_lc(x2, x1, k);
    x2 = __funnelshift_lc(x3, x2, k);
    x3 = __funnelshift_lc(0u, x3, k);
    used += k;
  };
  // "11": no intervals; "1" and a 0: one residual segment, whose count follows
  const uint32_t cl = 2u * (31u - __clz(d + 1u)) + 1u;  // gamma(d)
  if (x0 >> 28 != 0xEu || (x0 << 3) >> (32u - cl) != d + 1u) return false;
  skip(3u + cl);
  uint32_t v = 0;
  bool ok = true;
#pragma unroll
  for (uint32_t u = 0; u < kPackedRegs; u++) {
    if (u < d) {
      const uint32_t h = min(__clz(x0), 8);  // zeta_3: 4 (h + 1) bits
      ok &= h < 8u;
      const uint32_t x = ((x0 << (h + 1u)) >> (29u - 3u * min(h, 7u))) - 1u;
      v = u == 0 ? zigzag_first(node, x) : v + x + 1u;
      skip(min(4u * (h + 1u), 32u));
    }
    id[u] = min(v, uint32_t(g.n - 1));  // a gather never leaves the labels
  }
  return ok && used == uint32_t(len) && uint64_t(v) < g.n;
}

// The most frequent of lab[0..d), d >= 1, the smallest on ties: a label's
// first occurrence counts all of them.
__device__ __forceinline__ uint32_t packed_mode(const uint32_t (&lab)[kPackedRegs], uint32_t d) {
  uint32_t bc = 0, bl = 0;
#pragma unroll
  for (uint32_t u = 0; u < kPackedRegs; u++) {
    uint32_t c = 1;
#pragma unroll
    for (uint32_t y = u + 1; y < kPackedRegs; y++) c += (y < d && lab[y] == lab[u]) ? 1u : 0u;
    if (u < d && (c > bc || (c == bc && lab[u] < bl))) {
      bc = c;
      bl = lab[u];
    }
  }
  return bl;
}

// One vertex of degree <= kPackedMaxDeg by one thread.  Up to kPackedRegs ids
// and labels stay in registers (road grid 1404^2, 2M vertices of degree <= 7:
// k_packed 72 -> 47 us); else the thread walks the vertex's bit range (or its
// small-CSR list) into its label slots, issues every label load at once and
// counts there (lane_mode).  Returns 1 when the label changed.
// lab: this thread's kPackedMaxDeg label slots (shared memory in k_packed,
// where a lane's slots start kPackedMaxDeg words after the previous lane's:
// an odd stride, so the 32 lanes' k-th slots fall in 32 different banks).
template <int kLoad>
__device__ __forceinline__ uint32_t packed_vertex(const IterArgs &a, const Ctx &c, uint32_t p, uint32_t *lab) {
  const DevGraph &g = a.g;
  // kLdFenced: the labels change between the caller's grid-wide barriers,
  // whose fences make plain loads see them (ld.global.nc would not)
  const auto load = [&](uint32_t i) { return kLoad == kLdFenced ? c.lab_in[i] : ld_label(c, i); };
  const uint32_t node = g.vertices[p];
  const uint32_t d = g.deg[p];
  const uint32_t old = load(node);
  if (d == 0) return 0;
  const bool cgr = p < g.n_c;
  const uint32_t *ids = cgr ? nullptr : g.small_nbr + g.small_off[p - g.n_c];
  uint32_t nl = old;
  bool done = false;
  if (d <= kPackedRegs) {
    uint32_t r[kPackedRegs];
    done = true;
    if (cgr) {
      done = packed_ids(g, p, node, d, r);
    } else {
#pragma unroll
      for (uint32_t u = 0; u < kPackedRegs; u++) r[u] = u < d ? __ldg(ids + u) : 0u;
    }
    if (done) {
#pragma unroll
      for (uint32_t u = 0; u < kPackedRegs; u++) r[u] = u < d ? load(r[u]) : 0u;
      nl = packed_mode(r, d);
    }
  }
  if (!done) {
    uint32_t k = 0;
    bool bad = d > kPackedMaxDeg;
    if (!bad && cgr) {
      const int64_t r = walk_vertex_buf<true>(g.words, g.offsets[p], g.offsets[p + 1], node, g.n, [&](uint32_t id) {
        if (k < kPackedMaxDeg) lab[k] = id;
        k++;
      });
      bad = r != int64_t(d);
    }
    if (bad) {
      set_error(a.err, kErrBadStream);
      return 0;
    }
    uint32_t lv[kPackedMaxDeg];
#pragma unroll
    for (uint32_t j = 0; j < kPackedMaxDeg; j++) lv[j] = j < d ? (cgr ? lab[j] : __ldg(ids + j)) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kPackedMaxDeg; j++) lv[j] = j < d ? load(lv[j]) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kPackedMaxDeg; j++)
      if (j < d) lab[j] = lv[j];
    nl = lane_mode(lab, d);
  }
  c.lab_out[node] = nl;
  return nl != old;
}

// V2 (several vertices per warp) at its limit for the tiny bucket: one lane
// per position (packed_vertex), 32 vertices per warp; the lanes share nothing
// but the count of changed labels.
__global__ void __launch_bounds__(kThreads) k_packed(IterArgs a) {
  // per thread kPackedMaxDeg label slots: a per-thread array indexed at run
  // time would live in local memory
  __shared__ uint32_t slab[kThreads * kPackedMaxDeg];
  const Ctx c = resolve(a);
  busy_mark(a, 3, false);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long changed = 0;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < a.n_packed; i += nw) {
    const long long t0 = clock64();
    const PackedChunk ch = a.packed[i];
    const uint32_t mine = lane < ch.np ? packed_vertex<kLdShared>(a, c, ch.p0 + lane, slab + threadIdx.x * kPackedMaxDeg) : 0u;
    changed += mine;
    const uint32_t sc = __reduce_add_sync(kFull, mine);
    if (lane == 0) {
      if (a.seg_changed && sc) atomicAdd(a.seg_changed + ch.seg, sc);
      if (a.seg_cycles)
        atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + ch.seg),
                  (unsigned long long)((clock64() - t0) * a.cw_packed));
    }
  }
  busy_mark(a, 3, true);
  flush_changed(c.changed, changed);
}

// Waits until every block of the launch has arrived for the k-th time (k from
// 1).  Bounded: when the others do not arrive, the error word is set and
// every block gives up.  The launch is cooperative, so all blocks are resident.
__device__ __forceinline__ bool grid_barrier(PackedLoop *lp, uint32_t k, uint64_t limit, uint32_t *err) {
  __shared__ uint32_t s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&lp->arrived, 1u);
    const volatile uint32_t *seen = &lp->arrived, *gone = &lp->gone;
    unsigned long long t0 = 0;
    bool ok = true;
    // the clock on one poll in 64: reading it on each took 0.25 us an iteration
    for (uint32_t polls = 1; *seen < k * gridDim.x; polls++) {
      if ((polls & 63u) && limit) continue;
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (*gone || now - t0 >= limit) {
        ok = false;
        break;
      }
    }
    if (!ok) {
      set_error(err, kErrTimeout);
      atomicExch(&lp->gone, 1u);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0u;
}

// Every iteration of a plan that is all k_packed chunks in one launch: a
// graph of two kernels per iteration costs about 10 us an iteration beside
// the work (road grid 64^2),
// a barrier of the resident blocks 2 to 3 (lpa_run, 20 iterations: 207 -> 120 us;
// 362^2: 261 -> 195 us).
// Iterations lp->it .. lp->stop - 1 (lp->early: until nothing changes); block 0
// leaves the number of the iteration after the last in lp->it_end.
__global__ void __launch_bounds__(kThreads) k_packed_loop(IterArgs a, PackedLoop *lp) {
  __shared__ uint32_t slab[kThreads * kPackedMaxDeg];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t first = lp->it, stop = lp->stop;
  const bool early = lp->early != 0u;
  const uint64_t limit = lp->wait_ns;
  uint32_t it = first;
  bool ok = true;
  while (it < stop) {
    Ctx c;
    c.it = it;
    c.lab_in = (it & 1u) ? a.labs1 : a.labs0;
    c.lab_out = (it & 1u) ? a.labs0 : a.labs1;
    c.changed = a.changed + it;
    c.coherent = false;
    unsigned long long changed = 0;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < a.n_packed; i += nw) {
      const PackedChunk ch = a.packed[i];
      const uint32_t mine =
          lane < ch.np ? packed_vertex<kLdFenced>(a, c, ch.p0 + lane, slab + threadIdx.x * kPackedMaxDeg) : 0u;
      changed += mine;
      if (a.seg_changed) {
        const uint32_t sc = __reduce_add_sync(kFull, mine);
        if (lane == 0 && sc) atomicAdd(a.seg_changed + ch.seg, sc);
      }
    }
    flush_changed(c.changed, changed);
    it++;
    if (!grid_barrier(lp, it - first, limit, a.err)) {
      ok = false;
      break;
    }
    if (early && *reinterpret_cast<volatile unsigned long long *>(c.changed) == 0ull) break;
  }
  if (ok && blockIdx.x == 0 && threadIdx.x == 0) lp->it_end = it;
}

cudaError_t occupancy_packed_loop(int *blocks) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_packed_loop, kThreads, 0);
}

cudaError_t launch_packed_loop(int grid, cudaStream_t s, IterArgs a, PackedLoop *lp) {
  void *args[] = {&a, &lp};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_packed_loop), dim3(grid), dim3(kThreads), args, 0, s);
}

// The pre-pass over the record groups: a lane per record.  Each lane decodes
// its segment's ids into the warp's staging window (its lane in the top bits,
// or in the owner byte beside it), then the warp gathers the window's labels
// with 8 loads per lane in flight and stores them, consecutive ids of a segment
// to consecutive addresses.
template <int kGather, bool kPack>
__device__ __forceinline__ void decode_records(const IterArgs &a, const Ctx &c, uint32_t *wst, uint8_t *wown,
                                               uint64_t keep_pol) {
  const DevGraph &g = a.g;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t hot = uint32_t(min(g.n, uint64_t(kHotIds)));
  const uint32_t nmax = uint32_t(g.n - 1);
  uint32_t *ctr = a.work + kWorkCounters * (a.it_dev ? c.it : 0u) + kWqRecs;
  const auto claim = [&]() {
    uint32_t x = 0;
    if (lane == 0) x = atomicAdd(ctr, 1u);
    return __shfl_sync(kFull, x, 0);
  };
  // the next claim is made before a group runs where every warp gets several,
  // else after it, so that no warp holds a group another could run
  const bool eager = a.n_rgroups > 4u * gridDim.x * kWarps;
  for (uint32_t gi = claim(), x = 0; gi < a.n_rgroups; gi = eager ? __shfl_sync(kFull, x, 0) : claim()) {
    const long long t0 = clock64();
    const RecGroup rg = a.rgroups[gi];
    if (eager && lane == 0) x = atomicAdd(ctr, 1u);
    bool bad = false;
    uint32_t cnt = 0, node = 0;
    uint64_t index = 0;
    BitReader r;
    if (lane < rg.n) {
      const uint4 rec = __ldcs(reinterpret_cast<const uint4 *>(a.recs) + rg.rec0 + lane);
      index = uint64_t((rec.y >> 12) & 0xFFu) << 32 | rec.z;
      cnt = (rec.y >> 20) & 0xFFu;
      node = rec.w;
      r.seek(g.words, uint64_t(rec.y & 0xFFFu) << 32 | rec.x);
      if (cnt == kSegCountMax) cnt = r.gamma(bad);
    }
    const uint32_t incl = warp_incl_scan(cnt, lane);
    const uint32_t excl = incl - cnt;
    const uint32_t tot = __shfl_sync(kFull, incl, 31);
    // window item f of lane l goes to sc[drel_l + f].  32 bits do: the records of
    // a group are neighbours in one plan segment, so their items lie within its
    // 16384 arcs, or, of a hub, within the group's own residual labels
    const uint64_t i0 = (uint64_t(__shfl_sync(kFull, uint32_t(index >> 32), 0)) << 32) |
                        __shfl_sync(kFull, uint32_t(index), 0);
    uint32_t *sb = i0 >= a.hub_arcs ? a.scratch_rest : a.scratch;  // a plan segment is all hub or none
    uint32_t *sc = sb + i0;
    const int32_t drel = int32_t(index - i0) - int32_t(excl);
    uint32_t done = 0, v = 0;
    for (uint32_t w0 = 0; w0 < tot; w0 += kDecodeWindow) {
      const uint32_t w1 = min(w0 + kDecodeWindow, tot);
      const uint32_t lim = excl + done < w1 ? min(cnt, w1 - excl) : done;
      uint32_t *dst = wst + (int32_t(excl) - int32_t(w0));
      const auto put = [&](uint32_t k, uint32_t id) {
        if constexpr (kPack) {
          dst[k] = (id & 0x07FFFFFFu) | (lane << 27);
        } else {
          dst[k] = id;
          wown[int32_t(excl) - int32_t(w0) + int32_t(k)] = uint8_t(lane);
        }
      };
      if (done == 0 && lim > 0) {
        v = zigzag_first(node, r.zeta3(bad));
        put(0, v);
        done = 1;
      }
      for (; done < lim; done++) {
        v += r.zeta3(bad) + 1u;
        put(done, v);
      }
      if (done) bad |= v > nmax;  // ids ascend: the last one is the largest
      __syncwarp();
      for (uint32_t f0 = w0; f0 < w1; f0 += 256) {
        uint32_t lv[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t f = f0 + 32u * u + lane;
          const uint32_t id = f < w1 ? min(kPack ? wst[f - w0] & 0x07FFFFFFu : wst[f - w0], nmax) : 0u;
          lv[u] = f >= w1 ? 0u
                  : (kGather == 2 || (kGather == 0 && id < hot)) ? __ldg(c.lab_in + id)
                                                                  : ld_cg_keep(c.lab_in + id, keep_pol);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t f = f0 + 32u * u + lane;
          const uint32_t ol = f < w1 ? (kPack ? wst[f - w0] >> 27 : wown[f - w0]) : 0u;
          const int32_t rel = __shfl_sync(kFull, drel, ol) + int32_t(f);
          if (f < w1) __stcs(sc + rel, lv[u]);
        }
      }
      __syncwarp();
    }
    if (__any_sync(kFull, bad) && lane == 0) set_error(a.err, kErrBadStream);
    if (a.seg_cycles && lane == 0)
      atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + rg.seg),
                (unsigned long long)((clock64() - t0) * a.cw_decode));
  }
}

// Two-pass variant, pass 1, in two parts: decode groups, then record groups
// (decode_records).  Where the handle has segment records those take the
// residual segments and the decode groups the interval segments alone; without
// them (streamed handles, no memory for the records, streams or scratches beyond
// a record's fields) the decode groups take both.
//
// Decode groups: every 256-bit segment is decoded by one lane, which writes the labels of its ids (not the ids) to
// the scratch, so pass 2 only counts.  A warp takes one decode group (32
// segments) at a time from the iteration's work queue (IterArgs::work slot
// kWqGroups, zeroed before the launch).  Lane l finds its position with a warp scan of the positions'
// segment counts and a 5-step search; the lanes of one position reserve their
// output range with one atomicAdd on the position's cursor, since the labels
// of a position may sit in any order.  No block barriers: warps run alone.
// kGather (lpa_tune.gather_cache) picks the cache path of the residual label
// reads: 1 all through L2 only (ld.global.cg), leaving L1 to the bitstream;
// 2 all through L1, which pays when a few hot labels take many of the reads;
// 0 the labels of the lowest kHotIds ids (BFS order puts the hubs there)
// through L1 and the rest through L2 only.  A hot set about the size of the
// L1 left beside the window wins: against the lowest n/64 ids (262,144 at
// R-MAT scale 24) 8192 took the pre-pass from 2.336 to 2.257 ms at scale 24
// and the copy-model iteration from 24.75 to 24.34 ms, scale 22 within
// 0.5 %; 4096 and 16384 measured the same as 8192 at scale 24.
//
// kStage (lpa_tune.stage_stream) moves each group's stream span (the words its
// segments read, DecodeGroup::w0/wn) ahead of its decode with the copy
// engine: 1 a bulk prefetch of the next group's span into L2
// (cp.async.bulk.prefetch.L2) while the warp decodes the current one; 2 a 1-D
// bulk copy of the next group's span into one of two shared-memory buffers of
// the warp (cp.async.bulk ... mbarrier::complete_tx, 16-byte aligned, no
// multicast), completed on that buffer's mbarrier with a bounded wait, so the
// copy of group k + 1 overlaps the decode of group k; the lanes then read
// their words from the buffer (words outside the copied span, if any, from
// the stream itself).  Record groups read the stream directly; a group of
// interval segments alone has the residual segments between them in its span,
// so with records the knob moves words that no lane reads: an iteration at R-MAT
// scale 22 takes 1055 / 1094 / 1364 us with 0 / 1 / 2, of a 4M-vertex copy
// model 691 / 737 / 1073, at scale 14 to 20 the same with 0 and 1 within 2 %.
//
// kPack (n <= 2^27, unstaged forms): a staged id carries its lane in its top
// 5 bits, so the window needs no owner bytes (one shared store per id fewer:
// pre-pass 2.45 -> 2.39 ms at R-MAT scale 24).
template <int kGather, int kStage, bool kPack>
__global__ void __launch_bounds__(kThreads, 4) k_decode_two_pass(IterArgs a) {
  __shared__ uint32_t stage[kWarps * kDecodeWindow];
  __shared__ uint8_t owner[kPack ? 1 : kWarps * kDecodeWindow];
  extern __shared__ __align__(16) uint32_t sspan[];  // kStage 2: kSpanSmemBytes of dynamic shared memory
  __shared__ uint64_t sbar[kStage == 2 ? kWarps * 2 : 1];
  using WS = typename std::conditional<kStage == 2, StagedWords, GWords>::type;
  const DevGraph &g = a.g;
  const Ctx c = resolve(a);
  const uint32_t hot = uint32_t(min(g.n, uint64_t(kHotIds)));  // kGather 0: ids below read through L1
  // label reads through L2 keep their lines there ahead of the scratch, which
  // is written with streaming stores (read once, by the count pass):
  // 4.417 -> 4.396 ms per iteration at R-MAT scale 24
  const uint64_t keep_pol = l2_evict_last_policy();
  busy_mark(a, 0, false);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  // Decode groups come from the iteration's work queue, group_claim at a
  // time, each warp's next claim made one ahead so that its atomic is off the
  // critical path.  A fixed grid-stride assignment left SMs idle for 28 % of
  // the kernel at R-MAT scale 22 (ncu: 0.66 ms of SM activity in a 0.92 ms
  // launch): groups whose interval segments expand thousands of ids finished
  // late on the warps that drew them.
  // With one group a claim (group_claim, group_base: a graph of few groups per warp)
  // every warp's first group is its own instead (warp w of block b takes group
  // w * gridDim.x + b, so that neighbouring groups, a hub's among them, start
  // on different SMs): when the first two claims came from the queue with 4
  // groups each, most warps had no work while the first ones ran 8 groups in
  // a row (pre-pass at R-MAT scale 16 / 18 / 20: 111 / 144 / 258 us, now 51 /
  // 82 / 168 us).
  uint32_t *gctr = a.work + kWorkCounters * (a.it_dev ? c.it : 0u) + kWqGroups;
  const auto claim = [&]() {
    uint32_t x = 0;
    if (lane == 0) x = a.group_base + atomicAdd(gctr, a.group_claim);
    return __shfl_sync(kFull, x, 0);
  };
  uint32_t gi = a.group_base ? warp * gridDim.x + blockIdx.x : claim();
  uint32_t ahead = claim(), cend = gi + a.group_claim;
  uint32_t *wspan = sspan + (kStage == 2 ? warp * 2 * kSpanWords : 0);
  uint64_t *wbar = sbar + (kStage == 2 ? warp * 2 : 0);
  uint32_t phase[2] = {0u, 0u};
  // the words [lo, lo + n) of group gi's span that buffer b receives
  const auto span_of = [&](const DecodeGroup &d, uint64_t &lo, uint32_t &n) {
    lo = d.w0 & ~uint64_t(3);
    const uint64_t hi = min(min(d.w0 + d.wn, a.wend), lo + kSpanWords);
    n = hi > lo ? uint32_t((hi - lo) & ~uint64_t(3)) : 0u;
  };
  const auto issue = [&](uint32_t gi, uint32_t b) {  // lane 0
    const DecodeGroup d = a.groups[gi];
    uint64_t lo;
    uint32_t n;
    span_of(d, lo, n);
    if (n) bulk_load(wspan + b * kSpanWords, g.words + lo, n * 4u, wbar + b);
    else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(wbar + b)) : "memory");
  };
  if (kStage == 2) {
    if (lane == 0) {
      mbar_init(wbar, 1u);
      mbar_init(wbar + 1, 1u);
    }
    fence_mbar_init();
    __syncwarp();
    if (lane == 0 && gi < a.n_groups) issue(gi, 0u);
  }
  // the group after gi: the next of its claim, else the first of the claim
  // made ahead (which then becomes the current claim)
  const auto advance = [&]() {
    if (gi + 1u < cend) {
      gi++;
    } else {
      gi = ahead;
      cend = ahead + a.group_claim;
      ahead = claim();
    }
  };
  for (uint32_t it = 0; gi < a.n_groups; it++, advance()) {
    const long long t0 = clock64();
    const DecodeGroup gd = a.groups[gi];
    const uint32_t b = it & 1u;
    const uint32_t gnext = gi + 1u < cend ? gi + 1u : ahead;
    WS src;
    if (kStage == 1) {
      if (lane == 0 && gnext < a.n_groups) {
        const DecodeGroup dn = a.groups[gnext];
        const uint64_t hi = min(dn.w0 + dn.wn, a.wend);
        if (hi > dn.w0) prefetch_l2(g.words + dn.w0, (hi - dn.w0) * 4);
      }
    }
    if constexpr (kStage == 2) {
      // the other buffer's last reader (the previous group) is done: it
      // receives the next group's span while this one is decoded
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && gnext < a.n_groups) issue(gnext, b ^ 1u);
      if (!__all_sync(kFull, mbar_wait(wbar + b, phase[b], kBulkWaitTries))) {
        if (lane == 0) set_error(a.err, kErrTimeout);
        // neither copy may still write the buffers when the warp leaves
        mbar_wait(wbar + b, phase[b], kBulkWaitTries);
        if (gnext < a.n_groups) mbar_wait(wbar + (b ^ 1u), phase[b ^ 1u], kBulkWaitTries);
        break;
      }
      phase[b] ^= 1u;
      uint64_t lo;
      uint32_t n;
      span_of(gd, lo, n);
      src = StagedWords{g.words, wspan + b * kSpanWords, lo, n};
    } else {
      src = GWords{g.words};
    }
    const uint32_t pk = gd.p0 + lane;
    uint4 ix = make_uint4(0u, 0u, 0u, 0u);
    if (pk < g.n_c) ix = a.pidx[pk];
    if (a.rgroups) ix.w = 0u;  // the residual segments have records
    uint32_t ns = ix.z + ix.w;
    if (lane == 0) ns = ns > gd.j0 ? ns - gd.j0 : 0u;
    const uint32_t incl = warp_incl_scan(ns, lane);
    const uint32_t total = min(__shfl_sync(kFull, incl, 31), min(gd.nlanes, 32u));
    // owner: the number of positions whose segments all precede this lane
    uint32_t o = 0;
#pragma unroll
    for (uint32_t st = 16; st; st >>= 1) {
      const uint32_t v = __shfl_sync(kFull, incl, o + st - 1);
      if (v <= lane) o += st;
    }
    const uint32_t os = o & 31u;
    const uint32_t run0 = __shfl_sync(kFull, incl - ns, os);  // first lane of this position's run
    const uint32_t run1 = min(__shfl_sync(kFull, incl, os), total);
    const uint32_t ibr = __shfl_sync(kFull, ix.x, os), rbr = __shfl_sync(kFull, ix.y, os);
    const uint32_t nsi = __shfl_sync(kFull, ix.z, os);
    const bool act = lane < total;
    const uint32_t p = gd.p0 + os;
    const uint32_t jj = lane - run0 + (os == 0 ? gd.j0 : 0u);
    const bool itv = jj < nsi;
    bool bad = false;
    uint32_t cnt = 0, items = 0, node = 0;
    uint64_t q = 0, end = 0;
    BitReaderT<WS> r;
    if (act) {
      const uint64_t o0 = g.offsets[p];
      end = g.offsets[p + 1];
      node = g.vertices[p];
      q = o0 + (itv ? uint64_t(ibr) + uint64_t(kSegBits) * jj : uint64_t(rbr) + uint64_t(kSegBits) * (jj - nsi));
      if (q >= end) {
        bad = true;
      } else {
        r.seek(src, q);
        cnt = r.gamma(bad);
        if (!itv) {
          items = cnt;
        } else {
          for (uint32_t k = 0; k < cnt && !bad; k++) {
            r.gamma(bad);
            items += r.gamma(bad) + kMinItv;
            if (r.pos() > end) bad = true;
          }
        }
      }
      if (bad) {
        cnt = 0;
        items = 0;
      }
    }
    // output ranges: exclusive scan of items within the position's run
    const uint32_t iincl = warp_incl_scan(items, lane);
    const uint32_t run_before = __shfl_sync(kFull, iincl - items, run0 & 31u);
    const uint32_t run_total = __shfl_sync(kFull, iincl, (run1 - 1) & 31u) - run_before;
    uint32_t base = 0;
    if (act && lane == run0 && run_total) base = atomicAdd(a.cursor + p, run_total);
    base = __shfl_sync(kFull, base, run0 & 31u);
      // residual segments, in windows of kDecodeWindow items of the group:
    // each lane decodes its own segment's ids into the warp's staging area
    // (its lane number beside each), then the warp gathers the window's
    // labels with 8 loads per lane in flight and stores them, consecutive
    // ids of a position to consecutive addresses
    uint64_t obase = 0;  // scratch index of this lane's first item
    bool coop = false;   // an interval segment, expanded by the whole warp below
    uint32_t ritems = 0;
    if (act) {
      const uint32_t d = g.deg[p];
      const uint32_t off = base + (iincl - items) - run_before;
      obase = a.arc_off[p] + off;
      if (uint64_t(off) + items > d) bad = true;
      else if (items && itv) coop = true;
      else ritems = items;
    }
    const uint32_t rincl = warp_incl_scan(ritems, lane);
    const uint32_t rexcl = rincl - ritems;
    const uint32_t rtot = __shfl_sync(kFull, rincl, 31);
    // window item f of lane l goes to scratch[gb + drel_l + f] (32-bit
    // arithmetic) when the group's residual items lie within 2^32 of lane 0's
    // first, which holds the lowest scratch index of the group
    const uint64_t gb = (uint64_t(__shfl_sync(kFull, uint32_t(obase >> 32), 0)) << 32) |
                        __shfl_sync(kFull, uint32_t(obase), 0);
    const bool rel32 = __all_sync(kFull, ritems == 0u || ((obase + ritems - gb) >> 32) == 0ull);
    const uint32_t drel = uint32_t(obase - gb) - rexcl;
    const uint32_t nmax = uint32_t(g.n - 1);
    uint32_t *wst = stage + warp * kDecodeWindow;
    uint8_t *wown = owner + (kPack ? 0u : warp * kDecodeWindow);
    uint32_t done = 0, v = 0;
    for (uint32_t w0 = 0; w0 < rtot; w0 += kDecodeWindow) {
      const uint32_t w1 = min(w0 + kDecodeWindow, rtot);
      // this lane's items up to `lim` fall in this window, item i at window
      // index rexcl + i - w0 (>= 0 for every item not yet written)
      const uint32_t lim = rexcl + done < w1 ? min(ritems, w1 - rexcl) : done;
      uint32_t *dst = wst + (int32_t(rexcl) - int32_t(w0));
      // staged: the id with its lane in the top bits (kPack: the id's low 27
      // bits, so the lane stays intact) or in the owner bytes; the gather
      // clamps it to n - 1, once per 32 ids rather than once per code
      const auto put = [&](uint32_t k, uint32_t id) {
        if constexpr (kPack) {
          dst[k] = (id & 0x07FFFFFFu) | (lane << 27);
        } else {
          dst[k] = id;
          wown[int32_t(rexcl) - int32_t(w0) + int32_t(k)] = uint8_t(lane);
        }
      };
      if (done == 0 && lim > 0) {
        v = zigzag_first(node, r.zeta3(bad));
        put(0, v);
        done = 1;
      }
      for (; done < lim; done++) {
        v += r.zeta3(bad) + 1u;
        put(done, v);
      }
      // a segment's ids ascend, so its last one is its largest: an id past
      // n - 1 reads label n - 1, and the error word reports the stream (its
      // end is checked once, below).  Clamping instead of testing every id
      // took the pre-pass from 2.49 to 2.45 ms at R-MAT scale 24.
      if (done) bad |= v > nmax;
      __syncwarp();
      for (uint32_t f0 = w0; f0 < w1; f0 += 256) {
        uint32_t lv[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t f = f0 + 32u * u + lane;
          const uint32_t id = f < w1 ? min(kPack ? wst[f - w0] & 0x07FFFFFFu : wst[f - w0], nmax) : 0u;
          lv[u] = f >= w1 ? 0u
                  : (kGather == 2 || (kGather == 0 && id < hot)) ? __ldg(c.lab_in + id)
                                                                  : ld_cg_keep(c.lab_in + id, keep_pol);
        }
        if (rel32) {
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const uint32_t f = f0 + 32u * u + lane;
            const uint32_t ol = f < w1 ? (kPack ? wst[f - w0] >> 27 : wown[f - w0]) : 0u;
            const uint32_t rel = __shfl_sync(kFull, drel, ol) + f;
            if (f < w1) __stcs(a.scratch + gb + rel, lv[u]);
          }
        } else {
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const uint32_t f = f0 + 32u * u + lane;
            const uint32_t ol = f < w1 ? (kPack ? wst[f - w0] >> 27 : wown[f - w0]) : 0u;
            const uint64_t ob = (uint64_t(__shfl_sync(kFull, uint32_t(obase >> 32), ol)) << 32) |
                                __shfl_sync(kFull, uint32_t(obase), ol);
            const uint32_t ox = __shfl_sync(kFull, rexcl, ol);
            if (f < w1) __stcs(a.scratch + ob + (f - ox), lv[u]);
          }
        }
      }
      __syncwarp();
    }
    if (ritems && r.pos() > end) bad = true;
    // interval segments: one (left, len) pair per lane per round, expanded by
    // the whole warp (an interval can hold thousands of ids).  A round with
    // few intervals copies them one after another, 32 consecutive ids per
    // step (a broadcast of the interval, then coalesced label loads and
    // stores); a round with many short ones expands their concatenation,
    // each lane taking every 32nd id and finding its interval by a search
    // over the lanes' scan.  The round takes the form with the lower
    // estimated instruction count: per interval 16 + 4 per 32 ids, against
    // 100 per 128 ids of the concatenation.  At R-MAT scale 24 (BFS order,
    // 2.5 % of compressed arcs in intervals) the one-at-a-time form took the
    // pre-pass from 3.14 to 2.93 ms.
    if (__any_sync(kFull, coop)) {
      uint32_t left_todo = 0, nextbase = 0, w = 0;
      if (coop) {
        r.seek(src, q);
        left_todo = r.gamma(bad);
      }
      // a section's last segment takes the overflow of the one before: < 512 bits, < 256 pairs
      for (uint32_t round = 0; round < 512u && __any_sync(kFull, coop && left_todo); round++) {
        uint32_t lo = 0, len = 0;
        if (coop && left_todo) {
          const uint32_t l = r.gamma(bad);
          lo = (left_todo == cnt) ? zigzag_first(node, l) : nextbase + l + 1u;
          len = r.gamma(bad) + kMinItv;
          left_todo--;
          if (bad || uint64_t(lo) + len > g.n || w + len > items) {
            bad = true;
            len = 0;
            left_todo = 0;
          }
          nextbase = lo + len;
        }
        const uint32_t incl2 = warp_incl_scan(len, lane);
        const uint32_t tot = __shfl_sync(kFull, incl2, 31);
        const uint64_t dst = obase + w;  // where this lane's interval goes
        const uint32_t solo = __reduce_add_sync(kFull, len ? 16u + 4u * ((len + 31u) >> 5) : 0u);
        if (solo <= 100u * ((tot + 127u) >> 7)) {
          for (uint32_t m = __ballot_sync(kFull, len != 0u); m; m &= m - 1u) {
            const uint32_t l = uint32_t(__ffs(m) - 1);
            const uint32_t lo_l = __shfl_sync(kFull, lo, l), len_l = __shfl_sync(kFull, len, l);
            const uint64_t d_l = (uint64_t(__shfl_sync(kFull, uint32_t(dst >> 32), l)) << 32) |
                                 __shfl_sync(kFull, uint32_t(dst), l);
            uint32_t k1 = 0;
            for (; k1 + 512 <= len_l; k1 += 512) {  // a long interval: 16 loads in flight
              uint32_t lv[16];
#pragma unroll
              for (int u = 0; u < 16; u++) lv[u] = ld_label(c, lo_l + k1 + 32u * u + lane);
#pragma unroll
              for (int u = 0; u < 16; u++) __stcs(a.scratch + d_l + k1 + 32u * u + lane, lv[u]);
            }
            for (uint32_t k0 = k1; k0 < len_l; k0 += 128) {
              uint32_t lv[4];
#pragma unroll
              for (int u = 0; u < 4; u++) {
                const uint32_t k = k0 + 32u * u + lane;
                lv[u] = k < len_l ? ld_label(c, lo_l + k) : 0u;
              }
#pragma unroll
              for (int u = 0; u < 4; u++) {
                const uint32_t k = k0 + 32u * u + lane;
                if (k < len_l) __stcs(a.scratch + d_l + k, lv[u]);
              }
            }
          }
        } else {
          // 4 ids per lane per step, their loads in flight together
          for (uint32_t i0 = 0; i0 < tot; i0 += 128) {
            uint32_t lv[4];
            uint64_t at[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const uint32_t i = i0 + 32u * u + lane;
              uint32_t ow = 0;
#pragma unroll
              for (uint32_t st = 16; st; st >>= 1) {
                const uint32_t v = __shfl_sync(kFull, incl2, ow + st - 1);
                if (v <= i) ow += st;
              }
              ow &= 31u;
              const uint32_t first = __shfl_sync(kFull, incl2 - len, ow);
              const uint32_t olo = __shfl_sync(kFull, lo, ow);
              const uint64_t odst = (uint64_t(__shfl_sync(kFull, uint32_t(dst >> 32), ow)) << 32) |
                                    __shfl_sync(kFull, uint32_t(dst), ow);
              at[u] = odst + (i - first);
              lv[u] = i < tot ? ld_label(c, olo + (i - first)) : 0u;
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
              if (i0 + 32u * u + lane < tot) __stcs(a.scratch + at[u], lv[u]);
          }
        }
        w += len;
      }
      if (coop && (left_todo || w != items)) bad = true;
    }
    if (__any_sync(kFull, bad) && lane == 0) set_error(a.err, kErrBadStream);
    if (a.seg_cycles && lane == 0)
      atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + gd.seg),
                (unsigned long long)((clock64() - t0) * a.cw_decode));
  }
  if (a.rgroups)
    decode_records<kGather, kPack>(a, c, stage + warp * kDecodeWindow, owner + (kPack ? 0u : warp * kDecodeWindow),
                                   keep_pol);
  busy_mark(a, 0, true);
}

#define LPA_DECODE_FORMS(G)                                           \
  template __global__ void k_decode_two_pass<G, 0, false>(IterArgs a); \
  template __global__ void k_decode_two_pass<G, 1, false>(IterArgs a); \
  template __global__ void k_decode_two_pass<G, 2, false>(IterArgs a); \
  template __global__ void k_decode_two_pass<G, 0, true>(IterArgs a);
LPA_DECODE_FORMS(0)
LPA_DECODE_FORMS(1)
LPA_DECODE_FORMS(2)
#undef LPA_DECODE_FORMS

namespace {

// f(ok, label) for this warp's share of src[0..d): 32U-label blocks w,
// w + nw, ... with U loads per lane in flight; warp-synchronous.  keep: the
// labels will be read again soon (keep them in L2).
template <bool keep, int U = 8, class F>
__device__ __forceinline__ void warp_stream(const uint32_t *__restrict__ src, uint32_t d, uint32_t w, uint32_t nw,
                                            F &&f, const uint32_t *__restrict__ labels = nullptr) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t b0 = w * 32u * U; b0 < d; b0 += nw * 32u * U) {
    uint32_t v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t k = b0 + 32u * u + lane;
      v[u] = k < d ? (keep ? __ldcg(src + k) : __ldcs(src + k)) : 0u;
    }
    if (labels) {  // src holds ids: gather their labels
#pragma unroll
      for (int u = 0; u < U; u++)
        v[u] = (b0 + 32u * u + lane < d) ? (v[u] < kHotIds ? __ldg(labels + v[u]) : __ldcg(labels + v[u])) : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t k = b0 + 32u * u;
      if (k < d) f(k + lane < d, v[u]);
    }
  }
}

// Exact counts of this warp's share of src[0..d) (32U-label blocks) into et,
// with a running argmax in best (the count insert() returns is the label's
// total so far).
template <int U = 8>
__device__ __forceinline__ void count_exact(const EpochTable &et, const uint32_t *__restrict__ src, uint32_t d,
                                            uint32_t w, uint32_t nw, uint64_t &best,
                                            const uint32_t *__restrict__ labels = nullptr) {
  const uint32_t lane = threadIdx.x & 31u;
  const auto ins = [&](uint32_t lab, uint32_t c) {
    const uint64_t cand = pack_best(et.insert(lab, c), lab);
    best = cand > best ? cand : best;
  };
  WarpRun run;
  warp_stream<false, U>(src, d, w, nw, [&](bool ok, uint32_t lab) {
    if (run.extend(ok, lab)) return;
    if (run.cnt && lane == 0) ins(run.lab, run.cnt);
    run.restart(ok, lab);
    const uint32_t c = warp_merge(ok, lab);
    if (c) ins(lab, c);
  }, labels);
  if (run.cnt && lane == 0) ins(run.lab, run.cnt);
}

// The sketch of src[0..d) by the whole block in 32U-label blocks: every
// occurrence added to the zeroed counters cms (a warp-uniform run of one
// label adds once), then the running argmax of the estimate over the labels
// in best.  Lanes are not folded by label first (warp_merge): the shared
// memory atomics absorb the conflicts of a mixed step for less than the
// folding costs (count pass 2.55 -> 2.40 ms at R-MAT scale 24).
template <int U>
__device__ __forceinline__ void sketch_count(uint32_t *cms, const uint32_t *__restrict__ src, uint32_t d, uint32_t lb,
                                             const uint32_t *seeds, uint64_t &best) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const auto add = [&](uint32_t lab, uint32_t w) {
#pragma unroll
    for (int r = 0; r < kCmsDepth; r++)
      atomicAdd(&cms[r * kCmsWidth + (cm_hash(r, (lab - lb) ^ seeds[r]) & (kCmsWidth - 1))], w);
  };
  WarpRun run;
  warp_stream<true, U>(src, d, warp, kWarps, [&](bool ok, uint32_t lab) {
    if (run.extend(ok, lab)) return;
    if (run.cnt && lane == 0) add(run.lab, run.cnt);
    run.restart(ok, lab);
    if (ok) add(lab, 1u);
  });
  if (run.cnt && lane == 0) add(run.lab, run.cnt);
  __syncthreads();
  // the estimate depends on the label only: a step whose labels all equal
  // the label evaluated last adds nothing
  uint32_t seen = kFull;
  warp_stream<false, U>(src, d, warp, kWarps, [&](bool ok, uint32_t lab) {
    const uint32_t okm = __ballot_sync(kFull, ok);
    if (__ballot_sync(kFull, ok && lab == seen) == okm) return;
    seen = __shfl_sync(kFull, lab, __ffs(okm) - 1);
    if (ok) {
      uint32_t est = kFull;
#pragma unroll
      for (int r = 0; r < kCmsDepth; r++) {
        const uint32_t v = cms[r * kCmsWidth + (cm_hash(r, (lab - lb) ^ seeds[r]) & (kCmsWidth - 1))];
        est = v < est ? v : est;
      }
      const uint64_t cand = pack_best(est, lab);
      best = cand > best ? cand : best;
    }
  });
}

// One share of an exact vertex's labels (BlockItem, kCountHash) by the whole
// block: best is this thread's best of them.  keys and counts (kCountBlockSlots
// each) and *top (the count of kTopLabel) are zero before and after.  A share whose labels overfill the table is
// counted again in 4, 16, ... parts of itself, told apart by further bits of
// the hash (a bijection of the label: 20 bits leave at most 4096 labels).
__device__ __noinline__ uint64_t count_share(uint32_t *keys, uint32_t *top, const uint32_t *src, uint32_t d,
                                             uint32_t lg, uint32_t share) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t *cnts = keys + kCountBlockSlots;
  uint64_t best = 0;
  for (uint32_t more = 0;; more += 2) {
    best = 0;
    bool full = false;
    for (uint32_t part = 0; part < 1u << more && !full; part++) {
      const uint32_t want = share << more | part, sh = 32u - lg - more;
      const auto ins = [&](uint32_t lab, uint32_t c) { full |= !table_add(keys, cnts, kCountBlockSlots, top, lab, c); };
      WarpRun run;
      warp_stream<true, 4>(src, d, warp, kWarps, [&](bool ok, uint32_t lab) {
        ok = ok && slot_hash(lab) >> sh == want;
        if (run.extend(ok, lab)) return;
        if (run.cnt && lane == 0) ins(run.lab, run.cnt);
        run.restart(ok, lab);
        const uint32_t c = warp_merge(ok, lab);
        if (c) ins(lab, c);
      });
      if (run.cnt && lane == 0) ins(run.lab, run.cnt);
      full = __syncthreads_or(full) != 0;
      for (uint32_t k = threadIdx.x; k < kCountBlockSlots; k += kThreads) {
        const uint32_t key = keys[k];
        if (key) {
          const uint64_t cand = pack_best(cnts[k], key - 1u);
          best = cand > best ? cand : best;
          keys[k] = 0u;
          cnts[k] = 0u;
        }
      }
      if (threadIdx.x == 0 && *top) {
        const uint64_t cand = pack_best(*top, kTopLabel);
        best = cand > best ? cand : best;
        *top = 0u;
      }
      __syncthreads();
    }
    if (!full) return best;
  }
}

// Block-wide maximum of v, returned to every thread.
__device__ __forceinline__ uint64_t block_max_u64(uint64_t v, uint64_t *red) {
  v = warp_max_u64(v);
  if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  uint64_t m = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) m = red[w] > m ? red[w] : m;
  __syncthreads();
  return m;
}

}  // namespace

// Two-pass variant, pass 2.  The labels of every compressed two-pass
// position sit in the scratch, so this kernel mostly streams and counts
// (positions of the small CSR gather their labels); it holds no staging area
// and runs five blocks per SM (48 registers).  Block items (largest first): exact
// degrees up to kCountBlockMax in a 4096-slot block table, or the sketch;
// the warps stream disjoint 256-label blocks of the vertex.  Warp items: up
// to 4 (tunable) positions of degree <= kCountWarpMax, one vertex at a time in the
// warp's 512-slot table, or up to 32 positions of degree <= 32, a lane each
// (few left to count: the warp one by one).  The same shared memory serves the warp tables, the block table
// (block epochs, disjoint from the warps') and the sketch (cleared before and
// after use).  Every position's pre-pass cursor is reset here.
// kHash: the plan has kCountHash items (the call in the item loop costs the
// others registers: 20 us of 430 at R-MAT scale 22).
template <bool kBulk, bool kHash>
__global__ void __launch_bounds__(kThreads, 5) k_count_two_pass(IterArgs a) {
  extern __shared__ __align__(128) unsigned long long cslots[];
  __shared__ uint64_t red[kWarps];
  __shared__ uint64_t s_bar[kWarps];  // per warp: completion of its bulk copies
  __shared__ uint32_t s_has, s_epoch;
  __shared__ uint32_t s_top;  // kHash: a share's count of kTopLabel
  __shared__ BlockItem s_bi;
  const DevGraph &g = a.g;
  const Ctx c = resolve(a);
  busy_mark(a, 1, false);
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  for (uint32_t i = t; i < kCountBlockSlots; i += kThreads) cslots[i] = 0ull;
  if (t == 0) s_epoch = kHeavyEpochFirst;
  if (lane == 0) mbar_init(s_bar + warp, 1u);
  fence_mbar_init();
  __syncthreads();
  uint32_t *qctr = a.work + kWorkCounters * (a.it_dev ? c.it : 0u) + kWqBlock;
  unsigned long long changed = 0;

  // Block items, claimed ahead: while the block works on item k, thread 0
  // holds item k + 1 (loaded) and the claim of item k + 2, so neither the
  // queue atomic nor the item load sits on an item's critical path.  An item
  // carries its position's degree, scratch offset and vertex id, so the
  // block streams labels at once.
  BlockItem nxt{};
  bool has_nxt = false;
  uint32_t claim = 0;
  if (t == 0) {
    const uint32_t c0 = atomicAdd(qctr, 1u), c1 = atomicAdd(qctr, 1u);
    s_has = c0 < a.n_cblock;
    if (s_has) s_bi = a.cblock[c0];
    has_nxt = c1 < a.n_cblock;
    if (has_nxt) nxt = a.cblock[c1];
    claim = atomicAdd(qctr, 1u);
    if (++s_epoch > 0xFFFFu) s_epoch = 0;
  }
  for (;;) {
    __syncthreads();
    if (!s_has) break;
    const BlockItem it = s_bi;
    if (s_epoch == 0) {  // the block epochs wrapped: clear the table once
      for (uint32_t k = t; k < kCountBlockSlots; k += kThreads) cslots[k] = 0ull;
      __syncthreads();
      if (t == 0) s_epoch = kHeavyEpochFirst;
    }
    __syncthreads();  // every thread holds the item before thread 0 moves on
    const long long t0 = clock64();
    const uint32_t d = it.d;
    const uint32_t *src = a.scratch + it.ao;
    uint32_t old = 0;
    if (t == 0) {
      a.cursor[it.p] = 0u;
      old = ld_label(c, it.node);  // needed at the end only
    }
    uint64_t best = 0;
    if ((it.kind & 15u) == kCountSketch) {
      uint32_t *cms = reinterpret_cast<uint32_t *>(cslots);
      for (uint32_t k = t; k < kCmsDepth * kCmsWidth; k += kThreads) cms[k] = 0u;
      const uint32_t lb = label_base(a, it.node);
      __syncthreads();
      sketch_count<8>(cms, src, d, lb, a.seeds, best);  // smaller blocks gain nothing at degree >= 1024
      best = block_max_u64(best, red);
      // leave no counter behind that a table could read as one of its slots
      for (uint32_t k = t; k < kCmsDepth * kCmsWidth; k += kThreads) cms[k] = 0u;
    } else if (kHash && (it.kind & 15u) == kCountHash) {
      uint32_t *keys = reinterpret_cast<uint32_t *>(cslots);
      for (uint32_t k = t; k < 2 * kCountBlockSlots; k += kThreads) keys[k] = 0u;
      if (t == 0) s_top = 0u;
      __syncthreads();
      best = block_max_u64(count_share(keys, &s_top, src, d, (it.kind >> 4) & 15u, it.kind >> 8), red);
    } else {
      // blocks small enough that every warp takes one: the critical path of
      // a vertex of 512..1024 labels is one block of 64 or 128, not 256
      const EpochTable et{cslots, min(next_pow2(2 * d), kCountBlockSlots), s_epoch};
      if (d <= 32u * 2u * kWarps) count_exact<2>(et, src, d, warp, kWarps, best);
      else if (d <= 32u * 4u * kWarps) count_exact<4>(et, src, d, warp, kWarps, best);
      else count_exact<8>(et, src, d, warp, kWarps, best);
      best = block_max_u64(best, red);
    }
    if (t == 0) {
      bool last = true;
      if (kHash && (it.kind & 15u) == kCountHash) {  // the last share to finish has the vertex's best
        HashSlot &hs = a.hash[it.slot];
        atomicMax(&hs.best, (unsigned long long)best);
        __threadfence();
        last = atomicAdd(&hs.done, 1u) + 1u == 1u << ((it.kind >> 4) & 15u);
        if (last) {
          __threadfence();
          best = atomicExch(&hs.best, 0ull);
          hs.done = 0u;
        }
      }
      if (last) {
        const uint32_t nl = d ? best_label(best) : old;
        c.lab_out[it.node] = nl;
        changed += (nl != old);
        if (a.seg_changed && nl != old) atomicAdd(a.seg_changed + it.seg, 1u);
      }
      if (a.seg_cycles)
        atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + it.seg),
                  (unsigned long long)((clock64() - t0) * kWarps * a.cw_count));
      // advance the pipeline (the block reads s_bi after the loop-top barrier)
      s_has = has_nxt;
      s_bi = nxt;
      has_nxt = claim < a.n_cblock;
      if (has_nxt) nxt = a.cblock[claim];
      claim = atomicAdd(qctr, 1u);
      if (++s_epoch > 0xFFFFu) s_epoch = 0;
    }
  }

  unsigned long long *wslots = cslots + warp * kCountWarpSlots;
  uint32_t wepoch = 0;
  uint32_t bphase = 0;  // parity of this warp's next bulk-copy phase
  bool stop = false;    // a bulk copy did not complete in time
  while (!stop) {
    uint32_t i0 = 0;
    const uint32_t claim = a.warp_claim ? a.warp_claim : 2u;
    if (lane == 0) i0 = atomicAdd(qctr + 1, claim);
    i0 = __shfl_sync(kFull, i0, 0);
    if (i0 >= a.n_cwarp) break;
    for (uint32_t q = i0; q < i0 + claim && q < a.n_cwarp; q++) {
      const CountItem it = a.cwarp[q];
      const long long t0 = clock64();
      uint32_t my_changed = 0;
      if (it.kind == kCountGroups) {
        const uint32_t p = it.p0 + lane;
        const bool valid = lane < it.np;
        const uint32_t node = valid ? g.vertices[p] : 0u;
        const uint32_t d = valid ? g.deg[p] : 0u;
        const uint32_t old = valid ? ld_label(c, node) : 0u;
        // compressed positions: labels in the scratch; the small CSR: ids
        const bool ids = it.p0 >= g.n_c;
        const uint64_t ao = !valid ? 0ull : (ids ? uint64_t(g.small_off[p - g.n_c]) : a.arc_off[p]);
        if (valid && !ids) a.cursor[p] = 0u;
        // the positions are consecutive, so their neighbours are one range:
        // stage all its labels in the warp's table memory first (8 loads per
        // lane in flight), then count from shared memory
        const uint32_t incl = warp_incl_scan(d, lane);
        const uint32_t excl = incl - d;
        const uint32_t total = __shfl_sync(kFull, incl, 31);  // <= 32 * 32
        const uint64_t ao0 = (uint64_t(__shfl_sync(kFull, uint32_t(ao >> 32), 0)) << 32) |
                             __shfl_sync(kFull, uint32_t(ao), 0);
        uint32_t *wstage = reinterpret_cast<uint32_t *>(wslots);
        // scratch labels: one bulk copy of the 16-byte-aligned bytes around
        // the range (the scratch is padded at its end), the labels then at
        // wstage[sh0..); the small CSR gathers ids
        const uint64_t b_lo = (ao0 * 4u) & ~15ull, b_hi = ((ao0 + total) * 4u + 15u) & ~15ull;
        const bool bulk = kBulk && !ids && total >= kBulkMinLabels && b_hi - b_lo <= kCountWarpSlots * 8u;
        const uint32_t sh0 = bulk ? uint32_t(ao0 & 3u) : 0u;
        if (bulk) {
          fence_proxy_async_smem();  // this lane's earlier accesses to wstage come first
          __syncwarp();
          if (lane == 0)
            bulk_load(wstage, reinterpret_cast<const char *>(a.scratch) + b_lo, uint32_t(b_hi - b_lo), s_bar + warp);
          if (!__all_sync(kFull, mbar_wait(s_bar + warp, bphase, kBulkWaitTries))) {
            if (lane == 0) set_error(a.err, kErrTimeout);
            mbar_wait(s_bar + warp, bphase, kBulkWaitTries);  // the copy still writes wstage
            stop = true;
            break;
          }
          bphase ^= 1u;
        } else {
          for (uint32_t k0 = 0; k0 < total; k0 += 256) {
            uint32_t v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
              const uint32_t kk = k0 + 32u * u + lane;
              v[u] = kk >= total ? 0u : (ids ? __ldg(g.small_nbr + ao0 + kk) : __ldcs(a.scratch + ao0 + kk));
            }
            if (ids) {
#pragma unroll
              for (int u = 0; u < 8; u++) v[u] = (k0 + 32u * u + lane < total) ? ld_label_gather(c, v[u]) : 0u;
            }
#pragma unroll
            for (int u = 0; u < 8; u++)
              if (k0 + 32u * u + lane < total) wstage[k0 + 32u * u + lane] = v[u];
          }
        }
        __syncwarp();
        const uint32_t *lbl = wstage + sh0;
        // a vertex whose labels are all equal takes that label: lane v checks
        // its own vertex; only the others are counted below
        bool mixed = false;
        const uint32_t first = (lane < it.np && d) ? lbl[excl] : 0u;
        for (uint32_t j = 1; j < d; j++) mixed |= lbl[excl + j] != first;
        if (lane < it.np && d && !mixed) {  // an isolated vertex keeps its label in both buffers
          c.lab_out[node] = first;
          my_changed += (first != old);
        }
        if (uint32_t rest = __ballot_sync(kFull, mixed)) {
          uint32_t nl = 0;
          if (one_by_one(__popc(rest), __reduce_max_sync(kFull, mixed ? d : 0u))) {
            for (; rest; rest &= rest - 1u) {
              const uint32_t l = uint32_t(__ffs(rest) - 1);
              const uint32_t x = warp_mode(lbl + __shfl_sync(kFull, excl, l), __shfl_sync(kFull, d, l));
              if (lane == l) nl = x;
            }
          } else if (mixed) {
            nl = lane_mode(lbl + excl, d);
          }
          if (mixed) {
            c.lab_out[node] = nl;
            my_changed += (nl != old);
          }
        }
        __syncwarp();
        // the staged labels must not read as table slots later
        const uint32_t used = bulk ? uint32_t(b_hi - b_lo) / 8u : (total + 1) / 2;
        for (uint32_t k2 = lane; k2 < used; k2 += 32) wslots[k2] = 0ull;
        __syncwarp();
      } else {
        // every vertex's metadata in one round of loads (lane j: vertex j)
        const bool vj = lane < it.np;
        const uint32_t nodej = vj ? g.vertices[it.p0 + lane] : 0u;
        const uint32_t dj = vj ? g.deg[it.p0 + lane] : 0u;
        const uint32_t oldj = vj ? ld_label(c, nodej) : 0u;
        for (uint32_t j = 0; j < it.np; j++) {
          const uint32_t p = it.p0 + j;
          const uint32_t node = __shfl_sync(kFull, nodej, j);
          const uint32_t d = __shfl_sync(kFull, dj, j);
          const uint32_t old = __shfl_sync(kFull, oldj, j);
          const bool ids = p >= g.n_c;
          if (lane == 0 && !ids) a.cursor[p] = 0u;
          if (++wepoch >= kLightEpochs) {
            for (uint32_t k = lane; k < kCountWarpSlots; k += 32) wslots[k] = 0ull;
            __syncwarp();
            wepoch = 1;
          }
          const EpochTable et{wslots, min(next_pow2(2 * d), kCountWarpSlots), wepoch};
          uint64_t bp = 0;
          if (ids) count_exact(et, g.small_nbr + g.small_off[p - g.n_c], d, 0, 1, bp, c.lab_in);
          // a vertex of at most 128 labels loads them in one step of four rows
          // rather than eight (count pass 2.26 -> 2.21 ms at R-MAT scale 24)
          else if (d <= 128) count_exact<4>(et, a.scratch + a.arc_off[p], d, 0, 1, bp);
          else count_exact(et, a.scratch + a.arc_off[p], d, 0, 1, bp);
          bp = warp_max_u64(bp);
          if (lane == 0) {
            const uint32_t nl = d ? best_label(bp) : old;
            c.lab_out[node] = nl;
            my_changed += (nl != old);
          }
          __syncwarp();
        }
      }
      changed += my_changed;
      const uint32_t sc = __reduce_add_sync(kFull, my_changed);
      if (lane == 0) {
        if (a.seg_changed && sc) atomicAdd(a.seg_changed + it.seg, sc);
        if (a.seg_cycles)
          atomicAdd(reinterpret_cast<unsigned long long *>(a.seg_cycles + it.seg),
                    (unsigned long long)((clock64() - t0) * a.cw_count));
      }
    }
  }
  busy_mark(a, 1, true);
  flush_changed(c.changed, changed);
}

template __global__ void k_count_two_pass<false, false>(IterArgs a);
template __global__ void k_count_two_pass<true, false>(IterArgs a);
template __global__ void k_count_two_pass<false, true>(IterArgs a);
template __global__ void k_count_two_pass<true, true>(IterArgs a);

template <int G>
static void launch_decode_form(uint32_t stage, int grid, cudaStream_t s, const IterArgs &a) {
  if (stage == 1) k_decode_two_pass<G, 1, false><<<grid, kThreads, 0, s>>>(a);
  else if (stage == 2) k_decode_two_pass<G, 2, false><<<grid, kThreads, kSpanSmemBytes, s>>>(a);
  else if (a.g.n <= (1ull << 27)) k_decode_two_pass<G, 0, true><<<grid, kThreads, 0, s>>>(a);
  else k_decode_two_pass<G, 0, false><<<grid, kThreads, 0, s>>>(a);
}

cudaError_t prepare_decode_two_pass() {
  cudaError_t e = cudaFuncSetAttribute(k_decode_two_pass<0, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(kSpanSmemBytes));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_decode_two_pass<1, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSpanSmemBytes));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_decode_two_pass<2, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSpanSmemBytes));
  return e;
}

void launch_decode_two_pass(uint32_t gather_cache, uint32_t stage, int grid, cudaStream_t s, const IterArgs &a) {
  if (gather_cache == 1) launch_decode_form<1>(stage, grid, s, a);
  else if (gather_cache == 2) launch_decode_form<2>(stage, grid, s, a);
  else launch_decode_form<0>(stage, grid, s, a);
}

void launch_count_two_pass(bool bulk, bool hash, int grid, cudaStream_t s, const IterArgs &a) {
  if (bulk && hash) k_count_two_pass<true, true><<<grid, kThreads, kCountSmemBytes, s>>>(a);
  else if (bulk) k_count_two_pass<true, false><<<grid, kThreads, kCountSmemBytes, s>>>(a);
  else if (hash) k_count_two_pass<false, true><<<grid, kThreads, kCountSmemBytes, s>>>(a);
  else k_count_two_pass<false, false><<<grid, kThreads, kCountSmemBytes, s>>>(a);
}

cudaError_t occupancy_decode_two_pass(int *blocks) {
  // the forms without shared-memory staging (the default); the staged form
  // holds more shared memory and runs fewer blocks per SM
  int b0 = 1, b1 = 1, b2 = 1;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_decode_two_pass<0, 0, false>, kThreads, 0);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_decode_two_pass<1, 0, false>, kThreads, 0);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, k_decode_two_pass<2, 0, false>, kThreads, 0);
  *blocks = b0 < b1 ? (b0 < b2 ? b0 : b2) : (b1 < b2 ? b1 : b2);
  return e;
}

cudaError_t occupancy_count_two_pass(int *blocks) {
  int b[4] = {1, 1, 1, 1};
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[0], k_count_two_pass<false, false>, kThreads, kCountSmemBytes);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[1], k_count_two_pass<true, false>, kThreads, kCountSmemBytes);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[2], k_count_two_pass<false, true>, kThreads, kCountSmemBytes);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b[3], k_count_two_pass<true, true>, kThreads, kCountSmemBytes);
  *blocks = min(min(b[0], b[1]), min(b[2], b[3]));
  return e;
}

__global__ void k_pos_index(DevGraph g, uint4 *pidx, uint32_t *err, uint64_t p_lo, uint64_t p_hi) {
  for (uint64_t p = p_lo + blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < p_hi;
       p += uint64_t(gridDim.x) * blockDim.x) {
    bool bad = false;
    const uint64_t o0 = g.offsets[p], end = g.offsets[p + 1];
    BitReader r;
    r.seek(g.words, o0);
    const uint32_t nsi = r.segcnt(bad);
    const uint64_t ibase = r.pos();
    uint64_t last = r.pos();
    if (!bad && nsi && ibase + uint64_t(kSegBits) * (nsi - 1) < end) {
      // only the last interval segment is unpadded: decode it to find its end
      BitReader q;
      q.seek(g.words, ibase + uint64_t(kSegBits) * (nsi - 1));
      const uint32_t cnt = q.gamma(bad);
      for (uint32_t k = 0; k < cnt && !bad && q.pos() <= end; k++) {
        q.gamma(bad);
        q.gamma(bad);
      }
      last = q.pos();
    } else if (nsi) {
      bad = true;
    }
    uint32_t nsr = 0;
    uint64_t rbase = last;
    if (!bad && last <= end) {
      r.seek(g.words, last);
      nsr = r.segcnt(bad);
      rbase = r.pos();
    }
    if (bad || rbase > end || rbase - o0 > 0xFFFFFFFFull || (nsr && rbase + uint64_t(kSegBits) * (nsr - 1) >= end)) {
      set_error(err, kErrBadStream);
      pidx[p] = make_uint4(0u, 0u, 0u, 0u);
    } else {
      pidx[p] = make_uint4(uint32_t(ibase - o0), uint32_t(rbase - o0), nsi, nsr);
    }
  }
}

__global__ void k_seg_numbers(const uint4 *pidx, const Seg *segs, const uint8_t *use, uint32_t nseg, uint64_t *nsr) {
  for (uint32_t s = blockIdx.x; s < nseg; s += gridDim.x) {
    if (!use[s]) continue;
    for (uint32_t p = segs[s].begin + threadIdx.x; p < segs[s].end; p += blockDim.x) nsr[p] = pidx[p].w;
  }
}

// A warp per position, a lane per segment.
__global__ void k_seg_counts(DevGraph g, const uint4 *pidx, const uint64_t *roff, uint64_t *cnt, uint32_t *err) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t p = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; p < g.n_c; p += nw) {
    const uint64_t r0 = roff[p];
    const uint32_t ns = uint32_t(roff[p + 1] - r0);
    for (uint32_t j = lane; j < ns; j += 32) {
      bool bad = false;
      BitReader r;
      r.seek(g.words, g.offsets[p] + pidx[p].y + uint64_t(kSegBits) * j);
      cnt[r0 + j] = r.gamma(bad);
      if (bad) set_error(err, kErrBadStream);
    }
  }
}

__global__ void k_seg_records(DevGraph g, const uint4 *pidx, const uint64_t *roff, const uint64_t *csum,
                              const uint64_t *index, SegRec *recs) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t p = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; p < g.n_c; p += nw) {
    const uint64_t r0 = roff[p], r1 = roff[p + 1];
    if (r0 == r1) continue;
    // the intervals' labels first, then the residuals' in stream order
    const uint64_t at = index[p] + g.deg[p] - (csum[r1] - csum[r0]) - csum[r0];
    for (uint64_t i = r0 + lane; i < r1; i += 32) {
      bool bad = false;
      BitReader r;
      uint64_t q = g.offsets[p] + pidx[p].y + uint64_t(kSegBits) * (i - r0);
      r.seek(g.words, q);
      uint32_t c = r.gamma(bad);
      if (c < kSegCountMax) q = r.pos();
      else c = kSegCountMax;
      const uint64_t o = at + csum[i];
      recs[i] = SegRec{uint32_t(q), uint32_t(q >> 32) | uint32_t(o >> 32) << 12 | c << 20, uint32_t(o), g.vertices[p]};
    }
  }
}

__global__ void k_seg_ranges(const Seg *segs, uint32_t nseg, const uint64_t *roff, uint32_t *seg_rec) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) {
    const uint64_t r0 = roff[segs[s].begin], r1 = roff[segs[s].end];
    seg_rec[2 * s] = uint32_t(r0);
    seg_rec[2 * s + 1] = uint32_t(r1 - r0);
  }
}

// The CSR by vertex id (lpa_decode_csr): where every vertex sits, its degree in
// row[v] (scanned by the caller), then the lists of the ids [v0, v1) into out,
// row[v0] first.  A vertex without a position has no neighbours.
__global__ void k_csr_inverse(const uint32_t *vertices, uint64_t n, uint32_t *pos) {
  for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < n; p += uint64_t(gridDim.x) * blockDim.x)
    pos[vertices[p]] = uint32_t(p);
}
__global__ void k_csr_degrees(const uint32_t *deg, const uint32_t *pos, uint64_t n, uint64_t *row) {
  for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v <= n; v += uint64_t(gridDim.x) * blockDim.x)
    row[v] = v < n && pos[v] != kFull ? deg[pos[v]] : 0u;
}
// A warp per 32 ids (warp_decode_batch: a lane per header, the residual
// segments spread over the lanes); ids with more than kCsrSplit arcs among
// them go to 8 warps, 4 ids each.  The lists keep the order of the stream,
// intervals first.
__global__ void __launch_bounds__(kThreads) k_decode_csr(DevGraph g, const uint32_t *pos, const uint64_t *row,
                                                         uint64_t v0, uint64_t v1, uint32_t *out, uint32_t *err) {
  constexpr uint32_t kCsrSplit = 4096;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5, chunks = (v1 - v0 + 31) / 32;
  const uint64_t r0 = row[v0];
  for (uint64_t w = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; w < chunks * 8; w += nw) {
    const uint64_t v = v0 + (w >> 3) * 32 + lane;
    const uint32_t share = uint32_t(w) & 7u;
    uint32_t p = kFull, d = 0, base = 0;
    if (v < v1) {
      p = pos[v];
      base = uint32_t(row[v] - r0);  // a chunk of ids holds fewer than 2^32 arcs
      d = uint32_t(row[v + 1] - row[v]);
    }
    if (__reduce_add_sync(kFull, min(d, kCsrSplit + 1)) > kCsrSplit) {
      if ((lane >> 2) != share) d = 0;
    } else if (share) {
      continue;
    }
    const bool cgr = d != 0 && p < g.n_c, small = d != 0 && p >= g.n_c;
    if (__any_sync(kFull, cgr) && !warp_decode_batch(g, out, cgr, p, uint32_t(v), cgr ? d : 0u, base, lane) && lane == 0)
      set_error(err, kErrBadStream);
    for (uint32_t m = __ballot_sync(kFull, small); m; m &= m - 1u) {
      const uint32_t l = uint32_t(__ffs(m) - 1);
      const uint32_t pl = __shfl_sync(kFull, p, l), dl = __shfl_sync(kFull, d, l), bl = __shfl_sync(kFull, base, l);
      const uint32_t *src = g.small_nbr + g.small_off[pl - g.n_c];
      for (uint32_t k = lane; k < dl; k += 32) out[bl + k] = __ldg(src + k);
    }
  }
}

// Decode positions into a CSR scratch (out-of-core handles).
__global__ void k_decode_positions(DecodeArgs a) {
  const DevGraph &g = a.g;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < a.n_pos;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t p = a.pos_list ? a.pos_list[i] : a.pos_begin + i;
    if (p >= g.n_c) continue;
    uint32_t *dst = a.out + a.arc_off[p];
    const uint64_t d = g.deg[p];
    uint64_t k = 0;
    const int64_t r = walk_vertex(GWords{g.words}, g.offsets[p], g.offsets[p + 1], g.vertices[p], g.n,
                                  [&](uint32_t id) {
                                    if (k < d) dst[k] = id;
                                    k++;
                                  });
    if (r != int64_t(d)) {
      set_error(a.err, kErrBadStream);
      for (uint64_t q = (r > 0 ? uint64_t(r) : 0); q < d; q++) dst[q] = g.vertices[p];
    }
  }
}

__global__ void k_degree_count(DevGraph g, uint32_t *deg_out, uint32_t *itv_out, uint32_t *err, uint64_t p_lo,
                               uint64_t p_hi, uint32_t *hubs, uint32_t *n_hubs) {
  for (uint64_t p = p_lo + blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < p_hi;
       p += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t d = 0, itv = 0;
    if (g.vertices[p] >= g.n) {
      set_error(err, kErrBadStream);
    } else if (p < g.n_c) {
      if (g.offsets[p + 1] - g.offsets[p] > kHubBits) {
        hubs[atomicAdd(n_hubs, 1u)] = uint32_t(p);
        continue;
      }
      int64_t iv = 0;
      const int64_t c = walk_vertex_buf(g.words, g.offsets[p], g.offsets[p + 1], g.vertices[p], g.n,
                                        [](uint32_t) {}, &iv);
      if (c < 0 || c > int64_t(0xFFFFFFFFll)) {
        set_error(err, kErrBadStream);
      } else {
        d = uint32_t(c);
        itv = uint32_t(iv);
      }
    } else {
      const uint32_t b = g.small_off[p - g.n_c], e = g.small_off[p - g.n_c + 1];
      if (e < b) {
        set_error(err, kErrBadStream);
      } else {
        d = e - b;
        for (uint32_t k = b; k < e; k++)
          if (g.small_nbr[k] >= g.n) {
            set_error(err, kErrBadStream);
            d = 0;
            break;
          }
      }
    }
    deg_out[p] = d;
    if (itv_out) itv_out[p] = itv;
  }
}

// The degree pass over the positions k_degree_count left out, a block each,
// its threads on the 256-bit segments: the same tests as walk_vertex_buf's,
// whose one thread walked the largest list for 4.5 ms at R-MAT scale 18.
__global__ void __launch_bounds__(kThreads) k_degree_hubs(DevGraph g, uint32_t *deg_out, uint32_t *itv_out,
                                                          uint32_t *err, const uint32_t *hubs, const uint32_t *n_hubs) {
  __shared__ unsigned long long s_base, s_last, s_items, s_itv;
  __shared__ uint32_t s_nseg;
  const uint32_t t = threadIdx.x;
  const uint32_t count = *n_hubs;
  for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
    const uint32_t p = hubs[i];
    const uint64_t end = g.offsets[p + 1];
    const uint32_t node = g.vertices[p];
    bool bad = false;
    // a section's header at bit `at`
    const auto header = [&](uint64_t at) {
      BitReader r;
      r.seek(g.words, at);
      const uint32_t ns = r.segcnt(bad);
      const uint64_t pos = r.pos();
      if (bad || pos > end || ns > (end - pos) / kSegBits + 1) bad = true;
      s_nseg = bad ? 0u : ns;
      s_base = s_last = pos;
    };
    if (t == 0) {
      header(g.offsets[p]);
      s_items = s_itv = 0;
    }
    __syncthreads();
    uint32_t nseg = s_nseg;
    uint64_t base = s_base;
    unsigned long long mine = 0;
    for (uint32_t j = t; j < nseg && !bad; j += kThreads) {
      const uint64_t q = base + uint64_t(kSegBits) * j;
      if (q >= end) {
        bad = true;
        break;
      }
      BitReader r;
      r.seek(g.words, q);
      const uint32_t cnt = r.gamma(bad);
      uint32_t left = 0;
      for (uint32_t c = 0; c < cnt && !bad; c++) {
        const uint32_t l = r.gamma(bad);
        left = (c == 0) ? zigzag_first(node, l) : left + l + 1u;
        const uint32_t len = r.gamma(bad) + kMinItv;
        if (bad || r.pos() > end || uint64_t(left) + len > g.n) {
          bad = true;
          break;
        }
        mine += len;
        left += len;
      }
      if (j == nseg - 1) s_last = r.pos();
    }
    if (mine) {
      atomicAdd(&s_items, mine);
      atomicAdd(&s_itv, mine);
    }
    __syncthreads();
    if (t == 0) header(s_last);
    __syncthreads();
    nseg = s_nseg;
    base = s_base;
    mine = 0;
    for (uint32_t j = t; j < nseg && !bad; j += kThreads) {
      const uint64_t q = base + uint64_t(kSegBits) * j;
      if (q >= end) {
        bad = true;
        break;
      }
      BitReader r;
      r.seek(g.words, q);
      const uint32_t cnt = r.gamma(bad);
      uint32_t v = 0;
      for (uint32_t c = 0; c < cnt && !bad; c++) {
        const uint32_t x = r.zeta3(bad);
        v = (c == 0) ? zigzag_first(node, x) : v + x + 1u;
        if (bad || r.pos() > end || uint64_t(v) >= g.n) {
          bad = true;
          break;
        }
        mine++;
      }
      if (j == nseg - 1) s_last = r.pos();
    }
    if (mine) atomicAdd(&s_items, mine);
    bad = __syncthreads_or(bad) != 0;
    if (t == 0) {
      const bool ok = !bad && s_last == end && s_items <= 0xFFFFFFFFull;
      if (!ok) set_error(err, kErrBadStream);
      deg_out[p] = ok ? uint32_t(s_items) : 0u;
      if (itv_out) itv_out[p] = ok ? uint32_t(s_itv) : 0u;
    }
    __syncthreads();  // the shared words are free for the next list
  }
}

__global__ void k_init_labels(uint32_t *a, uint32_t *b, uint64_t n) {
  for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < n; v += uint64_t(gridDim.x) * blockDim.x) {
    a[v] = uint32_t(v);
    b[v] = uint32_t(v);
  }
}

#include "noalloc_kernels.cuh"  // kernels of lpa_iterate_noalloc

}  // namespace lpa_dev
