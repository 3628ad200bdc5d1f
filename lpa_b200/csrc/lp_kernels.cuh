// Label-propagation kernels: launch-argument structs and kernel declarations.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace lpa_dev {

// Kernel variants (all produce identical labels).
enum Variant : int {
  kVarWarp = 0,     // V1: lane-per-vertex decode, warp-per-vertex counting (deg <= kV1MaxDeg)
  kVarPacked = 1,   // V2: lane-per-vertex decode, several vertices per warp counting (deg <= 32)
  kVarBlock = 2,    // V3: block per vertex, segment-parallel decode, block table / sketch
  kVarTwoPass = 3,  // V4: a decode pass writes a CSR scratch; counting reads it
  kNumVariants = 4,
  kVarPackedLanes = 5  // batch plans only: V2 on a tiny segment, one thread per position (packed_vertex)
};

constexpr int kThreads = 256;             // threads per block of the iteration kernel
constexpr int kWarps = kThreads / 32;
constexpr uint32_t kStage = 8192;         // staged ids/labels per block (1024 per warp)
constexpr uint32_t kTableSlots = 8192;    // 64-bit exact-count slots per block (1024 per warp)
constexpr uint32_t kWarpStage = kStage / kWarps;
constexpr uint32_t kWarpSlots = kTableSlots / kWarps;
constexpr uint32_t kV1MaxDeg = kWarpSlots - 1;         // 1023: a warp's table holds every distinct label
constexpr uint32_t kV2MaxDeg = 32;
constexpr uint32_t kBlockMaxSmemDeg = kTableSlots / 2; // exact degrees counted in shared memory (<= 4095)

constexpr uint32_t kLightSlots = 512;                  // 64-bit slots per warp of k_light
constexpr size_t kLightSmemBytes = size_t(kWarps) * (kLightSlots * 8 + kWarpStage * 4);

// dynamic shared memory of the iteration kernel
constexpr size_t kSmemBytes = size_t(kStage) * 4 + size_t(kTableSlots) * 8;

struct Seg {
  uint32_t begin, end;  // positions [begin, end)
};

// A work item with the device range it will read, so a warp or block can
// prefetch items it has claimed but not started.  Heavy: one segment by a
// block; light: positions [p0, p0 + np) of a segment by a warp, as many as one
// batch of its staging area takes (32 positions, kWarpStage labels).
struct WorkItem {
  uint32_t seg;
  uint32_t pf_bytes;   // bytes of the range to prefetch
  uint64_t pf_addr;    // device address of the range (bitstream bits, small-CSR ids or scratch ids)
  uint32_t p0, np;
};

// Work of the two-pass pre-pass: nlanes (<= 32) consecutive segments of the
// positions p0, p0 + 1, ..., starting at segment j0 of p0 (interval segments
// first, then residual ones) and spanning at most 32 positions.  seg is the
// plan segment its cycles are booked to.
struct DecodeGroup {
  uint32_t p0, j0, nlanes, seg;
  uint64_t w0;      // the stream words its segments read: [w0, w0 + wn)
  uint32_t wn, pad;
};
// staged ids per warp of the pre-pass: 1024 (32 KB per block with the lane in
// the ids' top bits) beat 768 by 1.5 %; 1280 and 1536 shrink L1 and lose 3 %
// and 13 % (R-MAT scale 24)
constexpr uint32_t kDecodeWindow = 1024;
// One residual segment of a resident handle, ready to decode (two-pass plans):
//   x         low 32 bits of q, the bit after the segment's count
//   y         q's next 12 bits | index's bits 32..39 << 12 | count << 20
//   z         low 32 bits of the scratch index of its first label
//   w         the vertex
// A count of kSegCountMax or more is stored as kSegCountMax with q at the count
// itself.  A group's setup without them (finding positions, reserving output,
// reading counts) was a quarter of the pre-pass's instructions: 588 -> 550 us
// at R-MAT scale 22, 82 -> 56 us at 18.  Records stay in stream order: sorted by
// count in windows of 64, 128 or 256, so that the lanes of a group finish
// together (lane use 66 -> 90 %), the pre-pass took 574, 583 and 588 us, because
// 32 neighbouring segments share 8 lines and 32 others do not; copying every
// lane's words to shared memory a group ahead took 852 us.  The index is into
// the hubs' scratch below IterArgs::hub_arcs, from there into the rest.
struct SegRec {
  uint32_t x, y, z, w;
};
constexpr uint32_t kSegCountMax = 255;
constexpr uint64_t kSegMaxBit = 1ull << 44, kSegMaxIndex = 1ull << 40;
struct RecGroup {
  uint32_t rec0, n, seg;  // records [rec0, rec0 + n), n <= 32, of one plan segment
};

// Decode groups a warp of the pre-pass claims from its work queue at once: 4
// where every resident warp gets several such claims, else 1, so that every
// warp gets work (a claim's atomic is off the critical path either way).
constexpr uint32_t kGroupClaim = 4;
inline uint32_t group_claim_for(uint32_t n_groups, int grid) {
  return uint64_t(n_groups) >= uint64_t(grid) * kWarps * kGroupClaim * 4 ? kGroupClaim : 1u;
}
// lpa_tune.gather_cache 0: the pre-pass reads the labels of ids below this
// through L1 (32 KB of labels), the others through L2 only
constexpr uint32_t kHotIds = 8192;
// lpa_tune.stage_stream 2: words of a group's stream span one shared-memory
// buffer holds (32 segments of < 512 bits plus their headers fit)
constexpr uint32_t kSpanWords = 576;
constexpr uint32_t kSpanSmemBytes = kWarps * 2 * kSpanWords * 4;  // its two buffers per warp (dynamic)

// Work of the two-pass count pass (k_count_two_pass): positions p0 ..
// p0 + np - 1, all of one kind, whose labels the pre-pass wrote to the
// scratch.  seg is the plan segment the cycles are booked to.
enum CountKind : uint32_t {
  kCountGroups = 0,  // np <= 32 positions of degree <= 32: a lane per vertex
  kCountWarp = 1,    // np <= 4 positions of degree <= kCountWarpMax: warp per vertex, 512-slot table
  kCountBlock = 2,   // one position, degree <= kCountBlockMax: block per vertex, 4096-slot table
  kCountSketch = 3,  // one position at or above the sketch threshold: block per vertex
  kCountHash = 4,    // one position, exact, degree <= PlanInputs::hash_max: a block per share of the labels' hashes
};
struct CountItem {
  uint32_t p0, np, seg, kind;
};
// A block item of the count pass, with everything its block needs up front.
struct BlockItem {
  uint64_t ao;              // scratch index of the position's labels (arc offset)
  uint32_t p, d, node;      // position, degree, vertex id
  uint32_t seg, kind, slot; // plan segment (cycles), kind (below), kCountHash: the vertex's HashSlot
};
// kind: CountKind in the low 4 bits; kCountHash: log2 of the shares in the
// next 4, the item's share in the rest.
// An exact vertex above the block table is counted share by share: the blocks
// of its items each stream all its labels (from L2) and count those whose hash
// falls to them, at most about kCountHashLoad different ones, in 4096 slots of
// shared memory; the last to finish holds the vertex's best.  One block with a
// table in global memory took 92 us (526 us with every label different) for
// the degree-25,057 hub of R-MAT scale 18.
constexpr uint32_t kCountHashLoad = 2048;
constexpr uint32_t kCountHashMaxLog = 12;
constexpr uint64_t kCountHashMax = uint64_t(kCountHashLoad) << kCountHashMaxLog;
// log2 of the shares of an exact vertex of degree d.
__host__ __device__ inline uint32_t hash_share_log(uint32_t d) {
  uint32_t lg = 1;
  while ((uint64_t(kCountHashLoad) << lg) < d) lg++;
  return lg;
}
// Shares read a vertex's labels once each, so their work grows with the square
// of the degree, where a table in global memory (k_iterate, one block a vertex)
// reads them once: the shares win by their blocks until a graph has many
// vertices of several 100,000 neighbours.  100 of degree 1M: 60 to 70 ms in
// shares, 6 (all labels equal) / 10 (zipf) / 38 (all different) in tables;
// 300 of 300,000: 28 to 35 against 5.5 / 9.9 / 38; 1000 of 100,000: 8.4 / 9.3
// / 23 against 3.0 / 8.4 / 27; 10 of 1M: 6.7 to 8 against 6.2 / 8.6 / 22.
// hash_share_limit (runtime.cu) weighs the two with these rates, in ns a label:
constexpr double kShareNs = 1.17e-3;      // a label read by one share, the whole GPU on it
constexpr double kTableLatencyNs = 8.0;   // a label counted by one block
constexpr double kTableNs = 0.1;          // a label, all blocks counting
constexpr double kTableMargin = 1.5;      // the tables have to be faster by this
struct HashSlot {
  unsigned long long best;  // pack_best over the finished shares
  uint32_t done, pad;       // finished shares
};
constexpr uint32_t kCountWarpSlots = 512;
constexpr uint32_t kCountWarpMax = kCountWarpSlots - 1;  // tables fill up to load 1 (triangular probing)
constexpr uint32_t kCountBlockSlots = kWarps * kCountWarpSlots;  // the warps' tables together
// with lpa_tune.bulk_stage, group items of the count pass with at least this
// many scratch labels are staged by one bulk copy (cp.async.bulk) instead of
// per-lane loads
constexpr uint32_t kBulkMinLabels = 64;
constexpr uint32_t kBulkWaitTries = 1u << 22;  // mbarrier try_wait attempts before a copy counts as lost
constexpr uint32_t kCountBlockMax = 2047;
constexpr uint32_t kCountSmemBytes = kCountBlockSlots * 8;        // 32 KB

// Work of k_packed: up to 32 consecutive positions of one plan segment whose
// degrees are all <= kPackedMaxDeg, one lane each.
struct PackedChunk {
  uint32_t p0, np, seg, pad;
};
constexpr uint32_t kPackedMaxDeg = 15;  // the tiny bucket (degree < 16)

constexpr int kBusyKernels = 4;  // kernels of an iteration with a busy span (IterArgs::ktime)

// Work-queue counters of one iteration (IterArgs::work + kWorkCounters *
// slot): k_iterate's heavy items, k_light's items, the count pass's block and
// warp items, the pre-pass's decode and record groups; the rest unused.
enum WorkCounter : int { kWqHeavy = 0, kWqLight, kWqBlock, kWqWarp, kWqGroups, kWqRecs, kWorkCounters = 8 };

struct IterArgs {
  DevGraph g;
  uint32_t *labs0, *labs1;      // the two label buffers
  uint32_t parity0;             // iteration 0 of this launch reads labs0 when 0, labs1 when 1
  const uint32_t *it_dev;       // device iteration counter (CUDA-graph loop), nullptr: 0
  unsigned long long *changed;  // changed counters, indexed by the iteration counter
  uint32_t *work;               // work-queue counters: kWorkCounters per iteration slot
  uint32_t *err;
  const Seg *segs;              // all segments
  const uint8_t *seg_var;       // variant per segment
  const WorkItem *heavy;        // block work items (one segment each), largest first
  uint32_t n_heavy;
  const WorkItem *light;        // warp work items
  uint32_t n_light;
  const DecodeGroup *groups;    // two-pass pre-pass work: 32 segments per group
  uint32_t n_groups;
  uint32_t group_claim;         // groups a warp claims at once (group_claim_for)
  uint32_t group_base;          // with one group a claim: the warps' own first groups, else 0
  const SegRec *recs;           // the residual segments of record groups
  const RecGroup *rgroups;      // nullptr: the decode groups cover the residual segments too
  uint32_t n_rgroups;
  uint32_t *scratch_rest;       // base of scratch indices from hub_arcs on, for recs
  uint64_t hub_arcs;
  const uint4 *pidx;            // per compressed position: {ibase - offset, rbase - offset, nseg_i, nseg_r}
  const BlockItem *cblock;      // count-pass block items (largest first)
  uint32_t n_cblock;
  HashSlot *hash;               // of the kCountHash vertices; zero between launches
  const CountItem *cwarp;
  uint32_t n_cwarp;
  uint32_t warp_claim;          // warp items a warp of the count pass claims at once
  const PackedChunk *packed;    // k_packed work
  uint32_t n_packed;
  uint32_t cw_packed;           // cost weight of a k_packed warp-cycle (as cw_iterate)
  uint32_t *cursor;             // per compressed position: labels written by the pre-pass (pass 2 resets)
  long long *seg_cycles;        // per-segment device cycles (nullptr: off)
  // weights of one warp-cycle of k_iterate / k_light / k_decode_two_pass /
  // k_count_two_pass in seg_cycles: 960 / (the kernel's resident warps per
  // SM), so a booked unit is the same share of an SM whichever kernel spent it
  uint32_t cw_iterate, cw_light, cw_decode, cw_count;
  // nullptr, or the busy span of each kernel of the iteration on the GPU's
  // clock (ns): ktime[k] = earliest warp start, ktime[kBusyKernels + k] =
  // latest warp end, k = 0 k_decode_two_pass, 1 k_count_two_pass, 2 k_iterate and k_light,
  // 3 k_packed
  unsigned long long *ktime;
  uint32_t *seg_changed;        // per-segment changed counts (nullptr: off)
  uint32_t cms_thr;             // 0: no sketch
  uint32_t seeds[kCmsDepth];
  // two-pass scratch: the neighbours of compressed position p at
  // scratch[arc_off[p]..), as labels in any order (k_decode_two_pass) or as
  // ids (scratch_labels == 0)
  uint32_t *scratch;
  const uint64_t *arc_off;
  uint32_t scratch_labels;      // 1: the scratch holds labels (the pre-pass), 0: ids
  // global exact-count tables for exact vertices above kBlockMaxSmemDeg
  uint32_t *gtab;
  uint32_t gtab_slots;          // slots per block (power of two), 0: none
  // graphs concatenated into one (a lockstep batch): graph k owns the vertex
  // ids [gbase[k], gbase[k + 1]); n_gbase = 0: one graph
  const uint32_t *gbase;
  uint32_t n_gbase;
  // stream words [0, wend) that bulk copies may read (a multiple of 4: the
  // copies move whole 16-byte units inside the stream's allocation)
  uint64_t wend;
};

// The id base of the graph that owns vertex `node`.  The sketch hashes a
// label relative to it, so a graph's sketch counts are those of the graph run
// alone; the exact paths compare labels only and need no base.
__device__ __forceinline__ uint32_t label_base(const IterArgs &a, uint32_t node) {
  if (a.n_gbase == 0) return 0u;
  uint32_t lo = 0, hi = a.n_gbase;  // gbase[lo] <= node < gbase[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(a.gbase + mid) <= node) lo = mid;
    else hi = mid;
  }
  return __ldg(a.gbase + lo);
}

__device__ __forceinline__ uint32_t iter_index(const IterArgs &a) { return a.it_dev ? *a.it_dev : 0u; }

// ---- many graphs in one persistent launch ------------------------------
struct BatchGraph {
  DevGraph g;
  uint32_t *labs0, *labs1;
  const Seg *segs;
  const uint8_t *seg_var;
  uint32_t nseg;
};

// Queue items: (graph << 44) | (iteration << 32) | segment.
constexpr unsigned long long kQueueEmpty = ~0ull;

struct BatchArgs {
  const BatchGraph *graphs;
  uint32_t ngraphs;
  unsigned long long *queue;      // ring of items
  uint32_t cap;                   // ring capacity (> items of one iteration of every graph)
  unsigned long long *head, *tail;
  uint32_t *active;               // graphs still running
  uint32_t *done_items;           // per graph: items finished in its current iteration
  unsigned long long *changed;    // per graph: changed count of its current iteration
  uint32_t *iters;                // per graph: iterations finished
  uint32_t *err;
  uint32_t max_iter;
  int early_exit;
  uint32_t cms_thr;
  uint32_t seeds[kCmsDepth];
  uint32_t *gtab;
  uint32_t gtab_slots;
  unsigned long long spin_limit;  // bound on the wait for an empty queue
};

__global__ void k_batch(BatchArgs b);
__global__ void k_batch_init(const BatchGraph *graphs, uint32_t ngraphs);

__global__ void k_iterate(IterArgs a);
__global__ void k_light(IterArgs a);
// allows k_light its shared memory; its resident blocks per SM
cudaError_t prepare_light(int *blocks);
// kGather: the cache path of the residual label reads (lpa_tune.gather_cache);
// kStage: the stream staging (lpa_tune.stage_stream); kPack: staged ids carry
// their lane (n <= 2^27, unstaged forms)
template <int kGather, int kStage, bool kPack>
__global__ void k_decode_two_pass(IterArgs a);
// V2 for tiny vertices: a lane per vertex.
__global__ void k_packed(IterArgs a);
// Two-pass variant, pass 2: counts the labels the pre-pass wrote.
// kBulk: group items staged by bulk copies (lpa_tune.bulk_stage); kHash: the
// plan has kCountHash items
template <bool kBulk, bool kHash>
__global__ void k_count_two_pass(IterArgs a);

// The template forms of the two-pass kernels are launched and sized only in
// the file that defines them (lp_kernels.cu):
// k_decode_two_pass<gather_cache, stage_stream, pack> on `grid` blocks of kThreads;
void launch_decode_two_pass(uint32_t gather_cache, uint32_t stage, int grid, cudaStream_t s, const IterArgs &a);
// k_count_two_pass<bulk, hash> on `grid` blocks of kThreads with kCountSmemBytes;
void launch_count_two_pass(bool bulk, bool hash, int grid, cudaStream_t s, const IterArgs &a);
// allows the stage_stream 2 forms their dynamic shared memory (once per device)
cudaError_t prepare_decode_two_pass();
// the fewest resident blocks per SM over each kernel's forms.
cudaError_t occupancy_decode_two_pass(int *blocks);
cudaError_t occupancy_count_two_pass(int *blocks);

// The iterations of a plan that is all k_packed chunks in one cooperative
// launch: iterations [it, stop), early: until nothing changes.
struct PackedLoop {
  uint32_t it, stop, early;
  uint32_t it_end;         // out: the iteration after the last
  uint32_t arrived, gone;  // the barrier's arrivals; a block that gave up
  uint64_t wait_ns;        // how long a block waits at the barrier before it gives up
};
// A block waits for the longest share of an iteration (below 1 ms) and for
// blocks that have no SM yet, as long as other streams' kernels hold it: a
// time on the GPU's clock, far above both, not a number of polls.
constexpr uint64_t kBarrierWaitNs = 60ull * 1000 * 1000 * 1000;
cudaError_t occupancy_packed_loop(int *blocks);
cudaError_t launch_packed_loop(int grid, cudaStream_t s, IterArgs a, PackedLoop *lp);

struct DecodeArgs {
  DevGraph g;
  const uint32_t *pos_list;  // positions to decode (nullptr: [pos_begin, pos_begin + n_pos))
  uint64_t n_pos;
  uint64_t pos_begin;
  const uint64_t *arc_off;   // output offsets by position
  uint32_t *out;             // ids
  uint32_t *err;
};
__global__ void k_decode_positions(DecodeArgs a);

__global__ void k_csr_inverse(const uint32_t *vertices, uint64_t n, uint32_t *pos);
__global__ void k_csr_degrees(const uint32_t *deg, const uint32_t *pos, uint64_t n, uint64_t *row);
__global__ void k_decode_csr(DevGraph g, const uint32_t *pos, const uint64_t *row, uint64_t v0, uint64_t v1,
                             uint32_t *out, uint32_t *err);

// Per compressed position: where its interval and residual sections'
// segments start (relative to its bit offset) and how many each has.
// Positions [p_lo, p_hi) (compressed ones only).
__global__ void k_pos_index(DevGraph g, uint4 *pidx, uint32_t *err, uint64_t p_lo, uint64_t p_hi);

// The segment records (SegRec) of the positions p with nsr[p] != 0 (the
// numbers of their residual segments; roff: their exclusive sum, n_c + 1):
// k_seg_counts writes every segment's count to cnt[roff[p] + j],
// k_seg_records the records, given the counts' exclusive sum csum and every
// position's scratch index, k_seg_ranges every plan segment's records.
__global__ void k_seg_numbers(const uint4 *pidx, const Seg *segs, const uint8_t *use, uint32_t nseg, uint64_t *nsr);
__global__ void k_seg_counts(DevGraph g, const uint4 *pidx, const uint64_t *roff, uint64_t *cnt, uint32_t *err);
__global__ void k_seg_records(DevGraph g, const uint4 *pidx, const uint64_t *roff, const uint64_t *csum,
                              const uint64_t *index, SegRec *recs);
__global__ void k_seg_ranges(const Seg *segs, uint32_t nseg, const uint64_t *roff, uint32_t *seg_rec);

// Degrees (and interval items) of positions [p_lo, p_hi), a thread each;
// positions of more than kHubBits go to hubs[0..*n_hubs) (room for every
// compressed position of the range) and are left to k_degree_hubs.
constexpr uint64_t kHubBits = 4096;
__global__ void k_degree_count(DevGraph g, uint32_t *deg_out, uint32_t *itv_out, uint32_t *err, uint64_t p_lo,
                               uint64_t p_hi, uint32_t *hubs, uint32_t *n_hubs);
__global__ void k_degree_hubs(DevGraph g, uint32_t *deg_out, uint32_t *itv_out, uint32_t *err, const uint32_t *hubs,
                              const uint32_t *n_hubs);
__global__ void k_init_labels(uint32_t *a, uint32_t *b, uint64_t n);

}  // namespace lpa_dev
