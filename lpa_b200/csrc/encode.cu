// GPU-side CGR encoder, byte-identical to lpa::cgr_encode (cgr_format.cpp),
// which restates the reference's CgrCompressor (src/compressor.cpp:306-515).
//
// Everything runs on the device: the position order (a stable
// partition by degree class), the prefix sums of the bit lengths and of the small lists (host
// loops over the vertices took 10 ms at R-MAT scale 20) and the per-vertex
// work, one warp per compressed position:
//   pass 1  splits the neighbour list, 32 ids a step, into residuals and
//           intervals (maximal runs of >= 4 consecutive ids), kept in a work
//           array in the vertex's own range (residuals from its front,
//           (left, end) pairs from its back; 4 ids or more make 2 words), then
//           plans both sections' 256-bit segments with the reference's rule (a
//           segment closes when gamma(cnt + 1) + its bits + the next item's
//           bits exceed 256; the final partial segment joins the last closed
//           one, unpadded): a warp scan of the items' bits finds how many fit.
//           It gives the vertex's bit length, its item and segment counts and
//           the interval section's length;
//   pass 2  finds the same segments again and writes each: the lanes place
//           their codes in the warp's shared words, which then go to the
//           stream.  Non-last segments sit at fixed 256-bit steps and the last
//           is known from pass 1, so every segment's position is known.
// Bound by the chain of segments of the largest vertex (each start depends on
// the segment before), about 300 cycles a segment.  One thread per position,
// walking its list alone, held the GPU for the largest vertex's every id: R-MAT
// scale 20 took 45 + 120 ms in the two passes (largest degree 64,612).
// Words shared with the neighbouring vertices are OR-ed atomically into a
// zeroed stream.  Only the reference's parameters (zeta k = 3, intervals of
// >= 4, 256-bit segments for both sections) are supported.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cstdint>
#include <numeric>
#include <stdexcept>
#include <string>
#include <vector>

#include "lpa/cgr_format.h"

namespace {

constexpr uint32_t kSegLen = 256;
constexpr uint32_t kMinItv = 4;

__device__ __forceinline__ int sig_bit(uint64_t x) { return 63 - __clzll(x); }  // x > 0
__device__ __forceinline__ uint32_t gamma_size(uint64_t x) { return 2u * uint32_t(sig_bit(x + 1)) + 1u; }
__device__ __forceinline__ uint32_t zeta3_size(uint64_t x) { return (uint32_t(sig_bit(x + 1)) / 3u + 1u) * 4u; }
__device__ __forceinline__ uint64_t int_2_nat(int64_t x) {
  return x >= 0 ? uint64_t(x) << 1 : uint64_t(-((x << 1) + 1));
}

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kEncThreads = 256;
constexpr uint32_t kEncWarps = kEncThreads / 32;
// shared words per warp of a segment being written: below 512 bits plus the
// longer count, from any bit of its first word
constexpr uint32_t kSegWords = 24;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, v, o);
    if (lane >= uint32_t(o)) v += t;
  }
  return v;
}

// Positions a warp takes from the work counter: the large ones (first in
// position order, a hub can hold a warp for long) one by one, the others
// kEncClaim at a time.
constexpr uint32_t kEncClaim = 8;
struct Claim {
  uint64_t p, e;
};
__device__ __forceinline__ Claim claim_positions(unsigned long long *ctr, uint64_t n_large, uint64_t n_c,
                                                 uint32_t lane) {
  unsigned long long u = 0;
  if (lane == 0) u = atomicAdd(ctr, 1ull);
  u = __shfl_sync(kFull, u, 0);
  Claim c;
  if (u < n_large) {
    c.p = u;
    c.e = u + 1;
  } else {
    c.p = n_large + (u - n_large) * kEncClaim;
    c.e = c.p + kEncClaim;
  }
  if (c.e > n_c) c.e = n_c;
  return c;
}

// The items of one section of a vertex in the work array.
struct Section {
  const uint32_t *t;  // residuals: ids from the front; intervals: from the back
  uint64_t deg, n;    // ids of the vertex, items of the section
  uint32_t node;
  bool itv;
  __device__ __forceinline__ uint32_t left(uint64_t k) const { return itv ? t[deg - 1 - 2 * k] : t[k]; }
  __device__ __forceinline__ uint32_t end(uint64_t k) const { return itv ? t[deg - 2 - 2 * k] : 0u; }
  // item k's code value as the first of a segment or after item k - 1, and
  // (intervals) its length code
  __device__ __forceinline__ void codes(uint64_t k, bool first, uint64_t &code, uint64_t &len) const {
    const uint32_t l = left(k);
    len = itv ? uint64_t(end(k)) - l - kMinItv + 1 : 0;  // end: the last id
    if (first) code = int_2_nat(int64_t(l) - int64_t(node));
    else code = itv ? uint64_t(l) - end(k - 1) - 2 : uint64_t(l) - left(k - 1) - 1;
  }
  __device__ __forceinline__ uint32_t bits(uint64_t code, uint64_t len) const {
    return itv ? gamma_size(code) + gamma_size(len) : zeta3_size(code);
  }
};

// The segment of the section that starts at item s: how many items fit it, and
// their bits without the count.  Called by all lanes, same result in each.
__device__ __forceinline__ uint32_t fit_segment(const Section &sec, uint64_t s, uint32_t lane, uint32_t &bits) {
  uint32_t sum = 0, cnt = 0;
  for (;;) {
    const uint64_t k = s + cnt + lane;
    const bool has = k < sec.n;
    uint32_t b = 0;
    if (has) {
      uint64_t code, len;
      sec.codes(k, k == s, code, len);
      b = sec.bits(code, len);
    }
    const uint32_t incl = sum + warp_incl_scan(b, lane);
    const uint32_t fits = __ballot_sync(kFull, has && gamma_size(uint64_t(cnt) + lane + 1) + incl <= kSegLen);
    const uint32_t f = __popc(fits);  // the bits grow with every item: a prefix fits
    if (f) sum = __shfl_sync(kFull, incl, f - 1);
    cnt += f;
    if (f < 32) break;
  }
  bits = sum;
  return cnt;
}

// Bits of items [s, e) all coded as gaps.
__device__ __forceinline__ uint64_t gap_bits(const Section &sec, uint64_t s, uint64_t e, uint32_t lane) {
  uint32_t mine = 0;
  for (uint64_t k = s + lane; k < e; k += 32) {
    uint64_t code, len;
    sec.codes(k, false, code, len);
    mine += sec.bits(code, len);
  }
  return __reduce_add_sync(kFull, mine);
}

// plan_segments (cgr_format.cpp): segments and bits after the section's header.
__device__ __forceinline__ void plan_section(const Section &sec, uint32_t lane, uint32_t &nseg, uint64_t &bits) {
  uint64_t s = 0, last_s = 0;
  uint32_t closed = 0, last_cnt = 0, last_bits = 0, b = 0, cnt = 0;
  for (;;) {
    cnt = fit_segment(sec, s, lane, b);
    if (s + cnt >= sec.n) break;  // the open tail
    last_s = s;
    last_cnt = cnt;
    last_bits = b;
    closed++;
    s += cnt;
  }
  if (closed == 0) {
    nseg = 1;
    bits = gamma_size(cnt) + b;
  } else {
    nseg = closed;
    const uint64_t tail = gap_bits(sec, last_s + last_cnt, sec.n, lane);
    bits = uint64_t(closed - 1) * kSegLen + gamma_size(sec.n - last_s) + last_bits + tail;
  }
}

// Bits of x that end right before bit `end` of the words w (MSB first).
__device__ __forceinline__ void or_bits(uint32_t *w, uint32_t end, uint64_t x) {
  const uint32_t k = (end - 1) >> 5, sh = 31u - ((end - 1) & 31u);
  const uint32_t a = uint32_t(x << sh), b = uint32_t(sh ? x >> (32 - sh) : x >> 32), c = sh ? uint32_t(x >> (64 - sh)) : 0u;
  if (a) atomicOr(w + k, a);
  if (b) atomicOr(w + k - 1, b);
  if (c) atomicOr(w + k - 2, c);
}

// gamma(x) at bit `at` of the zeroed stream, by one thread.
__device__ __forceinline__ uint64_t put_gamma(uint32_t *words, uint64_t nwords, uint64_t at, uint64_t x, bool &bad) {
  const uint64_t end = at + gamma_size(x);
  if ((end + 31) / 32 > nwords) {
    bad = true;
    return end;
  }
  const uint64_t base = at >> 5;
  or_bits(words + base, uint32_t(end - base * 32), x + 1);
  return end;
}

// The segment of items [s, s + cnt) at bit `at`: gamma(cnt), the first item
// coded against the node, the rest as gaps.  buf: kSegWords zeroed shared
// words of the warp, left zeroed.  Returns the segment's end.
__device__ __forceinline__ uint64_t write_segment(const Section &sec, uint64_t s, uint32_t cnt, uint64_t at,
                                                  uint32_t *buf, uint32_t *words, uint64_t nwords, uint32_t lane,
                                                  bool &bad) {
  const uint32_t off = uint32_t(at) & 31u;
  uint32_t end = off + gamma_size(cnt);
  if (lane == 0) or_bits(buf, end, uint64_t(cnt) + 1);
  for (uint32_t j0 = 0; j0 < cnt; j0 += 32) {
    const uint32_t j = j0 + lane;
    uint64_t code = 0, len = 0;
    uint32_t b = 0;
    if (j < cnt) {
      sec.codes(s + j, j == 0, code, len);
      b = sec.bits(code, len);
    }
    const uint32_t incl = warp_incl_scan(b, lane);
    const uint32_t e = end + incl;
    if (b && e <= kSegWords * 32) {
      if (sec.itv) {
        or_bits(buf, e - gamma_size(len), code + 1);
        or_bits(buf, e, len + 1);
      } else {  // h zeros, a one, the 3 (h + 1) bits of code + 1
        or_bits(buf, e, (1ull << (b / 4 * 3)) | (code + 1));
      }
    }
    end += __shfl_sync(kFull, incl, 31);
  }
  __syncwarp();
  const uint64_t w0 = at >> 5;
  const uint32_t nw = (end + 31) / 32;
  if (nw > kSegWords || w0 + nw > nwords) {
    bad = true;
  } else if (lane < nw) {
    // the first and last words are shared with what lies beside the segment
    const uint32_t x = buf[lane];
    if (lane == 0 || lane == nw - 1) {
      if (x) atomicOr(words + w0 + lane, x);
    } else {
      words[w0 + lane] = x;
    }
  }
  __syncwarp();
  if (lane < kSegWords) buf[lane] = 0u;
  __syncwarp();
  return at - off + end;
}

__device__ __forceinline__ uint64_t write_section(const Section &sec, uint64_t base, uint32_t nseg, uint32_t *buf,
                                                  uint32_t *words, uint64_t nwords, uint32_t lane, bool &bad) {
  uint64_t s = 0, end = base;
  for (uint32_t k = 0; k < nseg && !bad; k++) {
    uint32_t b;
    const uint32_t cnt = k + 1 < nseg ? fit_segment(sec, s, lane, b) : uint32_t(sec.n - s);
    end = write_segment(sec, s, cnt, base + uint64_t(k) * kSegLen, buf, words, nwords, lane, bad);
    s += cnt;
  }
  return end;
}

struct EncodeArgs {
  const uint64_t *row;
  const uint32_t *clm, *vertices;
  uint32_t *work;           // one word per arc: the split lists
  uint64_t n_c, n_large;
  uint64_t *bits, *itv_bits;
  uint32_t *nseg_i, *nseg_r, *nres, *nitv;
  unsigned long long *ctr;  // work counter
  uint32_t *err;
};

// Pass 1: per compressed position its split lists, its bit length and the
// numbers pass 2 needs (item and segment counts, interval section length
// after its header).
__global__ void __launch_bounds__(kEncThreads) k_encode_size(EncodeArgs a) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  for (;;) {
    const Claim c = claim_positions(a.ctr, a.n_large, a.n_c, lane);
    if (c.p >= a.n_c) break;
    for (uint64_t i = c.p; i < c.e; i++) {
      const uint32_t v = a.vertices[i];
      const uint32_t *nb = a.clm + a.row[v];
      uint32_t *t = a.work + a.row[v];
      const uint64_t deg = a.row[v + 1] - a.row[v];
      // cons bit j: id j continues the run of id j - 1.  An id belongs to an
      // interval when three continuations in a row touch it.
      uint32_t cur = lane < deg ? nb[lane] : 0u, cons_before = 0;
      uint64_t nr = 0, ns = 0, ne = 0;
      bool bad = false;
      const auto cons_of = [&](uint32_t x, uint32_t left, uint64_t k) {
        const uint32_t up = __shfl_up_sync(kFull, x, 1);
        const uint32_t prev = lane ? up : left;
        const bool has = k < deg && k > 0;
        bad |= has && x <= prev;  // the gap codes need strictly ascending lists
        return __ballot_sync(kFull, has && uint64_t(prev) + 1 == uint64_t(x));
      };
      uint32_t cons = cons_of(cur, 0u, lane);
      for (uint64_t k0 = 0; k0 < deg; k0 += 32) {
        const uint64_t k = k0 + lane, kn = k + 32;
        const uint32_t nxt = kn < deg ? nb[kn] : 0u;
        const uint32_t cons_next = cons_of(nxt, __shfl_sync(kFull, cur, 31), kn);
        // bit 4 + j: id k0 + j
        const uint64_t x = (uint64_t(cons_before >> 28)) | (uint64_t(cons) << 4) | (uint64_t(cons_next & 15u) << 36);
        const uint64_t t3 = x & (x >> 1) & (x >> 2);
        const uint32_t in = uint32_t(((t3 >> 1) | t3 | (t3 << 1) | (t3 << 2)) >> 4);
        const uint32_t valid = deg - k0 >= 32 ? kFull : (1u << uint32_t(deg - k0)) - 1u;
        const uint32_t res = ~in & valid, starts = in & ~cons & valid, ends = in & ~uint32_t(x >> 5) & valid;
        if ((res >> lane) & 1u) t[nr + __popc(res & lt)] = cur;
        if ((starts >> lane) & 1u) t[deg - 1 - 2 * (ns + __popc(starts & lt))] = cur;
        if ((ends >> lane) & 1u) t[deg - 2 - 2 * (ne + __popc(ends & lt))] = cur;
        nr += __popc(res);
        ns += __popc(starts);
        ne += __popc(ends);
        cons_before = cons;
        cons = cons_next;
        cur = nxt;
      }
      if (__any_sync(kFull, bad)) {
        if (lane == 0) atomicOr(a.err, 1u);
        continue;
      }
      __syncwarp();  // the lists are read by other lanes below
      uint32_t nsi, nsr;
      uint64_t bi, br;
      plan_section(Section{t, deg, ns, v, true}, lane, nsi, bi);
      plan_section(Section{t, deg, nr, v, false}, lane, nsr, br);
      if (lane == 0) {
        a.nres[i] = uint32_t(nr);
        a.nitv[i] = uint32_t(ns);
        a.nseg_i[i] = nsi;
        a.nseg_r[i] = nsr;
        a.itv_bits[i] = bi;
        a.bits[i] = gamma_size(nsi - 1) + bi + gamma_size(nsr - 1) + br;
      }
    }
  }
}

// Pass 2: writes every compressed position at its offset.
__global__ void __launch_bounds__(kEncThreads) k_encode_write(EncodeArgs a, const uint64_t *offsets, uint32_t *words,
                                                              uint64_t nwords) {
  __shared__ uint32_t sbuf[kEncWarps * kSegWords];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t *buf = sbuf + (threadIdx.x >> 5) * kSegWords;
  if (lane < kSegWords) buf[lane] = 0u;
  __syncwarp();
  for (;;) {
    const Claim c = claim_positions(a.ctr, a.n_large, a.n_c, lane);
    if (c.p >= a.n_c) break;
    for (uint64_t i = c.p; i < c.e; i++) {
      const uint32_t v = a.vertices[i];
      const uint32_t *t = a.work + a.row[v];
      const uint64_t deg = a.row[v + 1] - a.row[v];
      const uint32_t nsi = a.nseg_i[i], nsr = a.nseg_r[i];
      const uint64_t ibase = offsets[i] + gamma_size(nsi - 1), rhead = ibase + a.itv_bits[i],
                     rbase = rhead + gamma_size(nsr - 1);
      bool bad = false;
      if (lane == 0) {
        put_gamma(words, nwords, offsets[i], nsi - 1, bad);
        put_gamma(words, nwords, rhead, nsr - 1, bad);
      }
      bad = __any_sync(kFull, bad);
      const uint64_t iend = write_section(Section{t, deg, a.nitv[i], v, true}, ibase, nsi, buf, words, nwords, lane, bad);
      const uint64_t rend = write_section(Section{t, deg, a.nres[i], v, false}, rbase, nsr, buf, words, nwords, lane, bad);
      if (lane == 0 && (bad || iend != rhead || rend != offsets[i + 1])) atomicOr(a.err, 2u);
    }
  }
}

// Position order.  k_class: a vertex's class as a one in the high (degree >=
// large) or low (>= small) half of x, 0 at n; after x's exclusive sum, whose
// halves count both classes before a vertex, k_place puts every vertex at its
// position: large by id, mid by id, small by id.
__global__ void k_class(const uint64_t *row, uint64_t n, uint64_t large, uint64_t small, uint64_t *x) {
  for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v <= n; v += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t d = v < n ? row[v + 1] - row[v] : 0u;
    x[v] = v == n ? 0u : d >= large ? 1ull << 32 : d >= small ? 1u : 0u;
  }
}
__global__ void k_place(const uint64_t *row, uint64_t n, uint64_t large, uint64_t small, const uint64_t *x,
                        uint32_t *vertices) {
  const uint64_t nl = x[n] >> 32, nm = x[n] & 0xFFFFFFFFull;
  for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < n; v += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t d = row[v + 1] - row[v], il = x[v] >> 32, im = x[v] & 0xFFFFFFFFull;
    vertices[d >= large ? il : d >= small ? nl + im : nl + nm + (v - il - im)] = uint32_t(v);
  }
}

// Degrees of ns vertices (and a 0 after them), for the scan to list offsets.
__global__ void k_small_degrees(const uint64_t *row, const uint32_t *vertices_small, uint64_t ns, uint64_t *deg) {
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k <= ns; k += uint64_t(gridDim.x) * blockDim.x)
    deg[k] = k < ns ? row[vertices_small[k] + 1] - row[vertices_small[k]] : 0u;
}

__global__ void k_narrow(const uint64_t *in, uint64_t n, uint32_t *out) {
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < n; k += uint64_t(gridDim.x) * blockDim.x)
    out[k] = uint32_t(in[k]);
}

// The small CSR: one warp copies each small vertex's list (lists are
// contiguous in both arrays, positions n_c.. in order).
__global__ void k_gather_small(const uint64_t *row, const uint32_t *clm, const uint32_t *vertices_small,
                               const uint32_t *small_off, uint64_t ns, uint32_t *small_graph) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t k = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; k < ns; k += nw) {
    const uint32_t v = vertices_small[k];
    const uint64_t b = row[v], d = row[v + 1] - b;
    uint32_t *dst = small_graph + small_off[k];
    for (uint64_t j = lane; j < d; j += 32) dst[j] = clm[b + j];
  }
}

void ck(cudaError_t e, const char *what) {
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw std::runtime_error(std::string("cgr_encode_gpu: ") + what + ": " + cudaGetErrorString(e));
  }
}

// Device arrays of one call, those added between two alloc()s in one allocation
// (400 us each above 1 MB, whatever the size).
class DevArrays {
 public:
  DevArrays() = default;
  DevArrays(const DevArrays &) = delete;
  DevArrays &operator=(const DevArrays &) = delete;
  ~DevArrays() {
    for (char *p : blocks_)
      if (p) cudaFree(p);
  }
  template <class T>
  void add(T **p, size_t count) {
    want_.push_back({reinterpret_cast<void **>(p), total_});
    total_ += (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
  }
  void alloc() {
    blocks_.push_back(nullptr);
    ck(cudaMalloc(&blocks_.back(), total_), "cudaMalloc");
    for (const Want &w : want_) *w.p = blocks_.back() + w.at;
    want_.clear();
    total_ = 0;
  }

 private:
  struct Want {
    void **p;
    size_t at;
  };
  std::vector<Want> want_;
  std::vector<char *> blocks_;
  size_t total_ = 0;
};

// Storage for n elements of an empty vector, in huge pages where the system has
// them: a fresh page costs more than copying into it (45 MB of stream: 14 ms in
// 4 KB pages, 6 in 2 MB ones, 7 in 4 KB pages touched by 16 threads).
template <class T>
void in_huge_pages(std::vector<T> &v, size_t n) {
  constexpr uintptr_t kHuge = 2u << 20;
  v.reserve(n);
  const uintptr_t p = reinterpret_cast<uintptr_t>(v.data());
  const uintptr_t a = (p + kHuge - 1) & ~(kHuge - 1), e = (p + n * sizeof(T)) & ~(kHuge - 1);
  if (e > a) madvise(reinterpret_cast<void *>(a), e - a, MADV_HUGEPAGE);  // advice: nothing to do when refused
}
template <class T>
void grow(std::vector<T> &v, size_t n) {
  in_huge_pages(v, n);
  v.resize(n);
}

}  // namespace

namespace lpa {

void cgr_encode_gpu(const CsrView &g, const CgrParams &p, int small_thresh, int large_thresh, CgrGraph &out,
                    int device) {
  if (p.zeta_k != 3 || p.min_itv_len != int(kMinItv) || p.itv_seg_len != int(kSegLen) ||
      p.res_seg_len != int(kSegLen))
    throw std::invalid_argument("cgr_encode_gpu: only the reference parameters (3, 4, 256, 256)");
  if (small_thresh < 0 || large_thresh < 0 || small_thresh > large_thresh)
    throw std::invalid_argument("cgr_encode_gpu: need 0 <= small_thresh <= large_thresh");
  if (g.n > 0xFFFFFFFFull) throw std::invalid_argument("cgr_encode_gpu: more than 2^32 vertices");
  ck(cudaSetDevice(device), "cudaSetDevice");
  const uint64_t n = g.n, m = n ? g.row[n] : 0;
  out = CgrGraph();
  out.n = n;
  out.small_thresh = small_thresh;
  out.large_thresh = large_thresh;
  int sms = 148;
  ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "attribute");
  const int wide = sms * 8;

  // position order: large by id, mid by id, small by id (as the host encoder)
  DevArrays mem;
  uint64_t *d_row, *d_class;
  uint32_t *d_vert;
  char *d_scan;
  size_t scan_bytes = 0;  // of the longest scan, over n + 1
  ck(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, static_cast<uint64_t *>(nullptr), static_cast<uint64_t *>(nullptr),
                                   n + 1), "scan");
  mem.add(&d_row, n + 1);
  mem.add(&d_class, n + 1);
  mem.add(&d_vert, n);
  mem.add(&d_scan, scan_bytes);
  mem.alloc();
  ck(cudaMemcpy(d_row, g.row, (n + 1) * 8, cudaMemcpyHostToDevice), "upload row");
  auto scan = [&](uint64_t *data, uint64_t count) {  // exclusive, in place; count <= n + 1
    size_t bytes = 0;
    ck(cub::DeviceScan::ExclusiveSum(nullptr, bytes, data, data, count), "scan");
    if (bytes > scan_bytes) throw std::runtime_error("cgr_encode_gpu: scan memory");
    ck(cub::DeviceScan::ExclusiveSum(d_scan, bytes, data, data, count), "scan");
  };
  k_class<<<wide, 256>>>(d_row, n, uint64_t(large_thresh), uint64_t(small_thresh), d_class);
  ck(cudaGetLastError(), "position order");
  scan(d_class, n + 1);
  uint64_t num = 0;
  ck(cudaMemcpy(&num, d_class + n, 8, cudaMemcpyDeviceToHost), "class sizes");
  out.n_large = num >> 32;
  const uint64_t n_c = out.n_c = out.n_large + (num & 0xFFFFFFFFull), ns = n - n_c;
  if (n_c == 0) {
    // nothing to compress: the small CSR is the graph (road grid 300^2 with
    // threshold 16: 2.5 ms by the passes below, 0.9 ms here)
    if (m > 0xFFFFFFFFull) throw std::invalid_argument("cgr_encode_gpu: small CSR exceeds 2^32 arcs");
    out.offsets.assign(1, 0);
    out.words.assign(4, 0u);
    if (n == 0) return;
    grow(out.vertices, n);
    std::iota(out.vertices.begin(), out.vertices.end(), 0u);
    grow(out.small_offset, n + 1);
    for (uint64_t v = 0; v <= n; v++) out.small_offset[v] = uint32_t(g.row[v] - g.row[0]);
    in_huge_pages(out.small_graph, m);
    out.small_graph.assign(g.clm + g.row[0], g.clm + m);
    return;
  }
  k_place<<<wide, 256>>>(d_row, n, uint64_t(large_thresh), uint64_t(small_thresh), d_class, d_vert);
  ck(cudaGetLastError(), "position order");
  const uint32_t *d_small = d_vert + n_c;

  // d_bits: the bit lengths, then their sums, the offsets
  uint32_t *d_clm, *d_work, *d_nsi, *d_nsr, *d_nres, *d_nitv, *d_so, *d_err;
  uint64_t *d_bits, *d_itv, *d_so64;
  unsigned long long *d_ctr;  // one per pass
  mem.add(&d_clm, m);
  mem.add(&d_work, m);
  mem.add(&d_bits, n_c + 1);
  mem.add(&d_itv, n_c);
  mem.add(&d_nsi, n_c);
  mem.add(&d_nsr, n_c);
  mem.add(&d_nres, n_c);
  mem.add(&d_nitv, n_c);
  mem.add(&d_so64, ns + 1);
  mem.add(&d_so, ns + 1);
  mem.add(&d_ctr, 2);
  mem.add(&d_err, 1);
  mem.alloc();
  if (m) ck(cudaMemcpy(d_clm, g.clm, m * 4, cudaMemcpyHostToDevice), "upload clm");
  ck(cudaMemset(d_ctr, 0, 16), "clear work counters");
  ck(cudaMemset(d_err, 0, 4), "clear error");
  EncodeArgs ea{d_row, d_clm, d_vert, d_work, n_c, out.n_large, d_bits, d_itv,
                d_nsi, d_nsr, d_nres, d_nitv, d_ctr, d_err};
  const int blocks = int(std::min<uint64_t>((n_c + kEncWarps - 1) / kEncWarps, uint64_t(wide)));
  k_encode_size<<<blocks, kEncThreads>>>(ea);
  ck(cudaGetLastError(), "size pass");
  grow(out.vertices, n);
  ck(cudaMemcpy(out.vertices.data(), d_vert, n * 4, cudaMemcpyDeviceToHost), "read positions");
  uint32_t err = 0;
  ck(cudaMemcpy(&err, d_err, 4, cudaMemcpyDeviceToHost), "read error");
  if (err) throw std::invalid_argument("cgr_encode_gpu: neighbour lists must be strictly ascending");
  ck(cudaMemset(d_bits + n_c, 0, 8), "clear last size");
  scan(d_bits, n_c + 1);
  ck(cudaMemcpy(&out.total_bits, d_bits + n_c, 8, cudaMemcpyDeviceToHost), "read total");
  // 4 zero words of tail, as the host encoder
  const uint64_t nwords = (out.total_bits + 31) / 32 + 4;
  // the small CSR's offsets (src/compressor.cpp:267-282)
  uint64_t acc = 0;
  if (ns) {
    k_small_degrees<<<wide, 256>>>(d_row, d_small, ns, d_so64);
    ck(cudaGetLastError(), "small offsets");
    scan(d_so64, ns + 1);
    k_narrow<<<wide, 256>>>(d_so64, ns + 1, d_so);
    ck(cudaGetLastError(), "small offsets");
    ck(cudaMemcpy(&acc, d_so64 + ns, 8, cudaMemcpyDeviceToHost), "read small total");
    if (acc > 0xFFFFFFFFull) throw std::invalid_argument("cgr_encode_gpu: small CSR exceeds 2^32 arcs");
  }
  uint32_t *d_words, *d_sg;
  mem.add(&d_words, nwords);
  mem.add(&d_sg, acc);
  mem.alloc();
  ck(cudaMemset(d_words, 0, nwords * 4), "clear stream");
  ea.ctr = d_ctr + 1;
  k_encode_write<<<blocks, kEncThreads>>>(ea, d_bits, d_words, nwords);
  ck(cudaGetLastError(), "write pass");
  if (acc) {
    k_gather_small<<<wide, 256>>>(d_row, d_clm, d_small, d_so, ns, d_sg);
    ck(cudaGetLastError(), "small CSR gather");
  }
  // the host's pages while the device writes
  grow(out.words, nwords);
  if (ns) grow(out.small_offset, ns + 1);
  if (acc) grow(out.small_graph, acc);
  out.offsets.resize(n_c + 1);
  ck(cudaMemcpy(out.offsets.data(), d_bits, (n_c + 1) * 8, cudaMemcpyDeviceToHost), "read offsets");
  ck(cudaMemcpy(&err, d_err, 4, cudaMemcpyDeviceToHost), "read error");
  if (err) throw std::runtime_error("cgr_encode_gpu: a vertex's bits did not end at its offset");
  ck(cudaMemcpy(out.words.data(), d_words, nwords * 4, cudaMemcpyDeviceToHost), "read stream");
  if (ns) ck(cudaMemcpy(out.small_offset.data(), d_so, (ns + 1) * 4, cudaMemcpyDeviceToHost), "read small offsets");
  if (acc) ck(cudaMemcpy(out.small_graph.data(), d_sg, acc * 4, cudaMemcpyDeviceToHost), "read small CSR");
}

}  // namespace lpa
