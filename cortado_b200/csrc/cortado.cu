// libcortado: the C-ABI drop-in for the reference's encode/decode path.
// Declarations and the reference entry point each function replaces are in
// include/cortado.h.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <float.h>
#include <stdint.h>
#include <string.h>

#include <mutex>

#include "../../include/cortado.h"
#include "decode.cuh"
#include "encode.cuh"
#include "kernels.cuh"

using namespace cortado;

// ================================================================== kernels
// Resident CTAs per SM each kernel is compiled for (register budget
// 65536 / (128 * n)); every kernel holds two 17 KiB buffers, so shared memory
// allows 6.  resi_recv runs 5 (a budget of 102 registers; it uses 96): at 80
// its client and residual words spill, and it measured 4.6% faster at 5;
// every other kernel measured slower at 5 (and the store 10% slower with a
// third buffer at 4).
#ifndef MINB_STORE
#define MINB_STORE 6
#endif
#ifndef MINB_REENC
#define MINB_REENC 6
#endif
#ifndef MINB_DEC
#define MINB_DEC 6
#endif
#ifndef MINB_RAPPLY
#define MINB_RAPPLY 5
#endif

namespace {

__device__ __forceinline__ Ctl& ctl_block() {
  extern __shared__ uint8_t smem_raw[];
  return *reinterpret_cast<Ctl*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
}

// The thread that issues a decoder's TMA loads and stores (warp 3, lane 0):
// bulk-store completion is tracked per thread, so the thread that loads over a
// buffer after a TMA store must be the one that issued the store.  (The encoders
// have no TMA stores; lane 0 of their warp 1 issues the loads.)
constexpr int TMA_TID = 96;

// Start of every CTA: takes its place in the launch's queue, reads the lookback
// epoch (both reads in flight together) and sets up the barriers.  The queue
// hands out the helper's place first (when there are at least two CTAs), then
// the chunks in order: a CTA's first place is also its first chunk, and every
// chunk handed out belongs to a CTA that is running.  Returns whether this CTA
// is the helper.  A chunk's barrier completes a phase per use: two arrivals by
// the prefetching lane (one before its loads are issued, one after the chunk's
// metadata and hand-copied bytes are written) plus the TMA bytes, so waiting on
// it also publishes the metadata.
__device__ __forceinline__ unsigned int next_place(const Sync& sy) {
  return atomicAdd(&sy.counter[0], 1u) - (gridDim.x < 2 ? 0u : 1u);
}
__device__ __forceinline__ bool begin_launch(Ctl& sm, const Sync& sy) {
  if (threadIdx.x == 0) {
    const unsigned int e = *(volatile unsigned int*)sy.epoch;
    const unsigned int p = next_place(sy);
    sm.epoch = e;
    sm.first = p;
    sm.pend[0].valid = sm.pend[1].valid = 0;
    sm.zeros = 0;
  }
  if (threadIdx.x == TMA_TID) {
    mbar_init(&sm.bar, 2);
    mbar_init(&sm.bar_src, 1);
    fence_mbar_init();
  }
  __syncthreads();
  return sm.first == 0xffffffffu;
}

// The last CTA out resets the chunk queue and advances the epoch for the next
// launch on this scratch; when the 16-bit epoch wraps it first clears the
// lookback words, so no word of an old launch can carry the new epoch.
// Returns the status word's value to the last CTA's thread 0 (else 0).
__device__ __forceinline__ unsigned int finish_launch(Ctl& sm, const Sync& sy, bool take_status = false) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    sm.is_last = atomicAdd(&sy.counter[1], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  unsigned int st = 0;
  if (sm.is_last) {
    const unsigned int e = sm.epoch;
    if (e == 65535u)
      for (long long i = threadIdx.x; i < sy.flags_cap; i += blockDim.x) {
        sy.flags[i] = 0;
        if (sy.offs) sy.offs[i] = 0;
      }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (take_status) st = atomicExch(sy.status, 0u);
      *sy.epoch = (e == 65535u) ? 0u : e + 1u;
      sy.counter[0] = 0;
      sy.counter[1] = 0;
      __threadfence();
    }
  }
  return st;
}

// Loads the float words of a chunk into a swizzled buffer (zero past nw).
__device__ __forceinline__ void load_plain_rows(uint32_t* buf, const uint8_t* src, long long c, int nw) {
  const uint32_t* g = reinterpret_cast<const uint32_t*>(src) + c * (long long)CW;
  for (int w = threadIdx.x; w < CW; w += blockDim.x) buf[swz(w)] = (w < nw) ? g[w] : 0u;
}

struct StreamHdr {
  long long n, chunks;
  int eb_e;
  bool ok;
};

__device__ __forceinline__ StreamHdr read_header(const uint8_t* s, long long bytes) {
  StreamHdr h;
  h.ok = bytes >= HDR;
  h.n = h.ok ? *reinterpret_cast<const long long*>(s) : 0;
  h.eb_e = h.ok ? *reinterpret_cast<const int*>(s + 8) : 1;
  h.ok = h.ok && h.n >= 0 && (h.n & 3) == 0 && h.eb_e >= 1 && h.eb_e <= 230;
  h.chunks = h.ok ? (h.n + CS - 1) / CS : 0;
  h.ok = h.ok && (HDR + 2 * h.chunks <= bytes);
  if (!h.ok) h.chunks = 0;
  return h;
}

// Writes a stream header (int64 N, int32 exponent, int32 0).
__device__ __forceinline__ void write_header(uint8_t* out, long long n, int eb_e) {
  *reinterpret_cast<long long*>(out) = n;
  reinterpret_cast<int*>(out)[2] = eb_e;
  reinterpret_cast<int*>(out)[3] = 0;
}

// ---- work sources: what a queue index means.
// One stream: the queue index is the chunk; arguments and tensor maps are the
// kernel's own parameters; a decoder's header was checked at kernel start.
struct SingleSrc {
  static constexpr bool batched = false;
  const OpArgs* a;
  const CUtensorMap* map_in;
  const CUtensorMap* map_out;
  long long total;
  StreamHdr h;
  Quant q1, q2;  // the bounds' quantizers (resolved on the device for NOA entry points)
  __device__ __forceinline__ void quant(int, Quant& x1, Quant& x2) const {
    x1 = q1;
    x2 = q2;
  }
  __device__ __forceinline__ int locate(long long g, int, long long& c) const {
    c = g;
    return 0;
  }
  __device__ __forceinline__ const OpArgs& args(int) const { return *a; }
  __device__ __forceinline__ const CUtensorMap* min(int) const { return map_in; }
  __device__ __forceinline__ const CUtensorMap* mout(int) const { return map_out; }
  __device__ __forceinline__ StreamHdr header(int) const { return h; }
  __device__ __forceinline__ int header_bad(int, const StreamHdr&) const { return 0; }
  // offset scanner over the stream's size table (one warp)
  __device__ __forceinline__ void scan(unsigned int epoch) const {
    if (total > 0) scan_offsets(a->sy.offs, epoch, reinterpret_cast<const uint16_t*>(a->in + HDR), h.chunks);
  }
};

// Many streams in one launch: the queue runs over the items' chunks back to
// back; each item has its own lookback words (Sync.flags offset by its chunk
// base), header and size.
struct __align__(64) BatchItem {
  CUtensorMap map_in;   // store: the floats; resi_recv: the client's floats
  CUtensorMap map_out;  // decoders: the output floats
  OpArgs a;             // a.sy.flags already offset to this item
  long long chunk_base; // first queue index of this item
  long long chunks;
};

template <int OP>
struct BatchSrc {
  static constexpr bool batched = true;
  const BatchItem* items;
  int n_items;
  long long total;
  // Item of queue index g, searched by the whole warp forward from `cur` (the
  // item of an earlier index of this CTA, or -1): 32 chunk bases per read.
  __device__ __forceinline__ int locate(long long g, int cur, long long& c) const {
    const int lane = threadIdx.x & 31;
    int lo = cur < 0 ? 0 : cur;
    while (true) {
      const int i = lo + lane;
      const bool le = i < n_items && items[i].chunk_base <= g;
      const int cnt = __popc(__ballot_sync(0xffffffffu, le));
      if (cnt < 32) {
        const int it = lo + cnt - 1;
        c = g - items[it].chunk_base;
        return it;
      }
      lo += 31;
    }
  }
  __device__ __forceinline__ const OpArgs& args(int i) const { return items[i].a; }
  __device__ __forceinline__ void quant(int i, Quant& x1, Quant& x2) const {
    x1 = items[i].a.q1;
    x2 = items[i].a.q2;
  }
  __device__ __forceinline__ const CUtensorMap* min(int i) const { return &items[i].map_in; }
  __device__ __forceinline__ const CUtensorMap* mout(int i) const { return &items[i].map_out; }
  __device__ __forceinline__ StreamHdr header(int i) const { return read_header(items[i].a.in, items[i].a.in_bytes); }
  // 0 = usable; 2 = size mismatch; 3 = corrupt header
  __device__ __forceinline__ int header_bad(int i, const StreamHdr& h) const {
    const OpArgs& a = items[i].a;
    if (!h.ok) return 3;
    const bool ok = h.n == a.n && (OP == OP_S2C || OP == OP_RESI || h.n <= a.out_cap);
    return ok ? 0 : 2;
  }
  // offset scanner over every usable item's size table, item after item
  __device__ __forceinline__ void scan(unsigned int epoch) const {
    for (int i = 0; i < n_items; i++) {
      const StreamHdr h = header(i);
      if (header_bad(i, h)) continue;
      scan_offsets(items[i].a.sy.offs, epoch, reinterpret_cast<const uint16_t*>(items[i].a.in + HDR), h.chunks);
    }
  }
};

__device__ __forceinline__ void tensormap_acquire(const CUtensorMap* m) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(m) : "memory");
}

// ---- the store's prefetch (its loader warp): finds the chunk of queue index g
// and starts its load into buffer t; lane 0 issues it.
struct WalkState {
  int item;                 // item of the last prefetched index (-1: none)
};

template <class Src>
__device__ __forceinline__ void prefetch_floats(Ctl& sm, int t, long long g, const Src& src, WalkState& ws) {
  const int lane = threadIdx.x & 31;
  StageMeta& m = sm.st[t];
  if (g >= src.total) {
    if (lane == 0) {
      m.g = g;
      mbar_arrive(&sm.bar);
      mbar_arrive(&sm.bar);
    }
    return;
  }
  long long c;
  const int item = src.locate(g, ws.item, c);
  const bool fresh = item != ws.item;
  ws.item = item;
  if (lane == 0) {
    const OpArgs& A = src.args(item);
    const int nw = (int)min((long long)CW, (A.n - c * CS) / 4);
    const bool tma = nw == CW && A.has_map_in;
    if (tma) {
      if (Src::batched && fresh) tensormap_acquire(src.min(item));
      fence_proxy_async();
      mbar_expect_tx(&sm.bar, CS);
      tma_load_rows(stage_buf(sm, t), src.min(item), (int)(c * 128), &sm.bar);
    } else {
      mbar_arrive(&sm.bar);
    }
    m.g = g;
    m.c = c;
    m.item = item;
    m.nw = nw;
    m.tma = tma;
    m.n = A.n;
    m.chunks = (A.n + CS - 1) / CS;
    m.bad = 0;
    mbar_arrive(&sm.bar);
  }
}

// ---- the three pipelined loops.  Each CTA dequeues chunk indices from the
// launch's queue; one warp (warp 1 of the encoders, warp 3 of the decoders)
// finds the chunk and starts its loads.  Decoders take their indices one
// iteration ahead, re-encoders once the present chunk has been expanded, the
// store once its planes are written; each loads the next chunk as soon as a
// buffer has room for it.
//
// Encoders publish a chunk's compressed size as soon as it is known and write
// its payload one iteration later (write_pending): by then every earlier chunk
// has published too, and the resolver CTA has usually turned the chunk's own
// lookback word into an inclusive prefix, so no CTA waits on its
// predecessors while it holds the SM.

// Requantization through floats (d_s2c.h:132-137, d_RESI_4.h:57-76): the
// stored bin (or, for a raw chunk, the float itself) -> float (iSQ) -> request
// bin (CQ), or residual = destination bin minus the request bin requantized
// to the destination bound.  For the words (bit k of m) that the shift form
// cannot take; the choice is per word, so one outlier no longer sends its
// warp's 1024 words down the slow path.  Out of line: such words are rare
// (lossless words, raw chunks), and inlining the integer forms 32 times over
// made the loop large enough to stall on instruction fetch.  The words are
// the calling thread's own row of a swizzled buffer (row_store before the
// call, row_load after): a pointer to the caller's register array would put
// that array in local memory for the whole loop.  Returns the word `before` the
// row's first, requantized as well when `slow_before`.
template <int OP>
__device__ __noinline__ uint32_t requant_words(uint32_t* buf, uint32_t m, uint32_t before, bool slow_before, bool raw,
                                               Quant qs, Quant q1, Quant q2) {
  auto requant = [&](uint32_t stored) -> uint32_t {
    const uint32_t x = raw ? stored : iq_dec(stored, qs);
    if (OP == OP_S2C) return cq_enc(x, q1);
    const uint32_t src_req = cq_enc(iq_dec(cq_enc(x, q1), q1), q2);
    return cq_enc(x, q2) - src_req;
  };
  const uint32_t base = 32u * threadIdx.x;
  for (; m; m &= m - 1) {
    const uint32_t w = swz(base + __ffs(m) - 1);
    buf[w] = requant(buf[w]);
  }
  return slow_before ? requant(before) : before;
}

// Resolves a pending chunk's output offset (one warp, before a barrier that
// publishes sm.payload_off) ...
template <class Src>
__device__ __forceinline__ void resolve_pending(Ctl& sm, const Src& src, const Pend& pd, int by = 0) {
  if ((threadIdx.x >> 5) == by && pd.valid) {
    const unsigned long long X = lookback_resolve(src.args(pd.item).sy, sm.epoch, pd.c, pd.csize);
    if ((threadIdx.x & 31) == 0) sm.payload_off = X;
  }
}
// ... and writes it out from its staging buffer (every thread, after that
// barrier).
// FLOATS: a raw chunk's payload is the input's floats, read again.
template <bool FLOATS, class Src>
__device__ __forceinline__ void write_pending(Ctl& sm, const Src& src, const Pend& pd, const uint32_t* st,
                                              const uint32_t* st_small) {
  if (!pd.valid) return;
  const OpArgs& Q = src.args(pd.item);
  const long long chunks = (Q.n + CS - 1) / CS;
  flush_staged<FLOATS>(sm, pd, st, st_small, FLOATS ? reinterpret_cast<const uint32_t*>(Q.in) + pd.c * (long long)CW : nullptr,
                       Q.out + HDR + 2 * chunks, reinterpret_cast<uint16_t*>(Q.out + HDR), Q.out_size, chunks);
}

// store (d_server_encode_kernel): floats -> SQ -> encode.  One buffer (A)
// receives a chunk's floats, which are quantized into registers, and then
// takes its planes and its payload; the other (B) holds the previous chunk's
// payload until it is flushed, and receives the next chunk after that.
// The previous chunk's offset is waited for only after this chunk's size has
// been published.  (Waiting before that, although the flush then hid the next
// load, let one late chunk hold up every CTA's next size: the wait took 3,000
// to 5,500 of 13,000 to 20,000 cycles per chunk.  256 MiB: nearly all zero bins
// 156 -> 137 us, sinusoids with noise 166 -> 160, dense 217 -> 214.)
template <class Src>
__device__ __forceinline__ void store_loop(Ctl& sm, const Src& src, const Sync& sy) {
  constexpr int LOADER = 1;  // the warp that takes chunks: its planes are rarely the dense ones
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  init_pack_table();  // (read after the loop's first barrier)
  WalkState ws{-1};
  auto take = [&]() -> unsigned int { return (warp == LOADER && lane == 0) ? next_place(sy) : 0u; };
  auto load = [&](int t, unsigned int g) {
    if (warp == LOADER) prefetch_floats(sm, t, __shfl_sync(0xffffffffu, g, 0), src, ws);
  };
  auto flush = [&](int t) { write_pending<true>(sm, src, sm.pend[t], stage_buf(sm, t), stage_buf(sm, t) + CW); };
  load(0, sm.first);
  int s = 0;  // this chunk's buffer and slots; also the barrier's phase
  for (;; s ^= 1) {
    if (!mbar_wait(&sm.bar, s, sy.timeout_ns)) latch(sy.status, DST_TIMEOUT);
    const StageMeta& m = sm.st[s];
    if (m.g >= src.total) break;
    uint32_t* A = stage_buf(sm, s);
    const OpArgs& A_ = src.args(m.item);
    if (!m.tma) {
      load_plain_rows(A, A_.in, m.c, m.nw);
      __syncthreads();
    }
    uint32_t v[32];
    row_load(A, tid, v);
    uint32_t prev0 = tid ? A[swz(32 * tid - 1)] : 0u;  // the word before (lane 0 uses it)
    bool some;  // this thread's bins (or the one before them) are not all zero
    {
      Quant q1, q2_unused;
      src.quant(m.item, q1, q2_unused);
      if (Src::batched && tid == 0 && m.c == 0) write_header(A_.out, A_.n, q1.eb_e);
      // the float form; a warp that holds lossless words (inf, NaN included)
      // chooses per word
      const FastQ fq = make_fastq(q1.eb_e);
      float amax = fabsf(__uint_as_float(prev0));
#pragma unroll
      for (int k = 0; k < 32; k += 2) amax = max3_abs(amax, __uint_as_float(v[k]), __uint_as_float(v[k + 1]));
      some = !(__fmul_rn(amax, fq.sc) < 1.0f);  // (bins truncate; true for inf and NaN)
      if (__all_sync(0xffffffffu, amax < __uint_as_float(fq.thr_bits))) {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = sq_fast(v[k], fq);
        prev0 = sq_fast(prev0, fq);
      } else {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = sq_mixed(v[k], fq, q1);
        prev0 = sq_mixed(prev0, fq, q1);
      }
    }
    unsigned int g = 0;
    Packer pz(0), pk(0);
    auto next = [&]() { g = take(); };
    auto near = [&](uint32_t) {
      // the next chunk's floats are loaded after the flush: bring them into L2
      if (!Src::batched && warp == LOADER && lane == 0 && (long long)g + 1 < src.total)
        prefetch_l2(A_.in + (long long)g * CS, CS);
    };
    bool enc = true;
    if (Src::batched) __syncthreads();  // (the batched form tells zeros behind the planes: 1% faster on other data)
    else enc = __syncthreads_or(some);
    // A has been read; the pending payload is complete
    if (enc) {
      encode_chunk<true, Src::batched>(sm, A_.sy, v, prev0, A, A, A + CW, m, sm.pend[s], pz, pk, []() {}, next, near);
    } else {  // all bins are zero: only the 2-byte trailer (128 MiB: 55 -> 51 us)
      if (tid == 0) {
        lookback_publish(A_.sy, sm.epoch, m.c, 2u);
        sm.pend[s] = Pend{m.c, m.item, m.nw, 2, 0, 1, 1};
        A[CW] = 4u * m.nw;
      }
      next();
      near(2u);
    }
    resolve_pending(sm, src, sm.pend[s ^ 1], LOADER);
    __syncthreads();  // the payload's full words are in place; sm.payload_off
    flush(s ^ 1);
    pz.finish(A);
    pk.finish(A);
    __syncthreads();  // the other buffer is free
    load(s ^ 1, g);
  }
  resolve_pending(sm, src, sm.pend[s ^ 1]);
  __syncthreads();
  flush(s ^ 1);
}

// ---- stream prefetch (one warp of a decoder or re-encoder CTA), in two parts.
// The payload offset comes from the launch's offset scanner (the prefix sum of
// the size table that the reference's decoders form per CTA, d_s2c.h:98-106).
constexpr int FEEDER = TMA_TID / 32;

// What resolve_stream leaves in flight (lane 0), until park_stream puts it into
// the metadata slot for issue_stream.
struct Ahead {
  unsigned long long off;  // the scanner's word
  int csize;
};

// First part, at the start of an iteration: finds the chunk of queue index g,
// fills its metadata slot and reads its size entry and offset word (not
// waited for here).
template <int OP, class Src>
__device__ __forceinline__ void resolve_stream(Ctl& sm, int t, long long g, const Src& src, WalkState& ws, Ahead& ah) {
  const int lane = threadIdx.x & 31;
  StageMeta& m = sm.st[t];
  ah.csize = 0;
  if (g >= src.total) {
    if (lane == 0) m.g = g;
    return;
  }
  long long c;
  const int item = src.locate(g, ws.item, c);
  const bool fresh = item != ws.item;
  ws.item = item;
  if (lane == 0) {
    const OpArgs& A = src.args(item);
    StreamHdr h;
    int bad;
    if (Src::batched && !fresh) {  // the header was read for the chunk before
      const StageMeta& o = sm.st[t ^ 1];
      h.n = o.n;
      h.chunks = o.chunks;
      h.eb_e = o.eb_e;
      bad = o.bad >= 2 ? o.bad : 0;
    } else {
      h = src.header(item);
      bad = src.header_bad(item, h);
      if (Src::batched) {
        tensormap_acquire(src.mout(item));
        tensormap_acquire(src.min(item));
      }
    }
    m.g = g;
    m.c = c;
    m.item = item;
    m.bad = bad;
    m.n = h.n;
    m.chunks = h.chunks;
    m.eb_e = h.eb_e;
    m.nw = CW;
    if (!bad) {
      m.nw = (int)min((long long)CW, (h.n - c * CS) / 4);
      ah.csize = reinterpret_cast<const uint16_t*>(A.in + HDR)[c];
      ah.off = ld_relaxed(&A.sy.offs[c]);
      const uint8_t* client = OP == OP_RAPPLY ? A.src : OP == OP_RESI ? A.client : nullptr;
      if (client && m.nw == CW) prefetch_l2(client + c * (long long)CS, CS);
    }
  }
  __syncwarp();
}

template <class Src>
__device__ __forceinline__ void park_stream(Ctl& sm, int t, const Src& src, const Ahead& ah) {
  StageMeta& m = sm.st[t];
  if ((threadIdx.x & 31) == 0) {
    m.off = ah.off;
    m.csize = ah.csize;
  }
  __syncwarp();
}

// Chunks below this one sum the sizes before them themselves when the scanner
// has not published their offset yet: at most eight loads per lane.
constexpr int OWN_SUM = 256;

// The offset of a payload that the scanner had not published when the chunk was
// taken (one warp).
__device__ __forceinline__ unsigned long long open_offset(const OpArgs& A, long long c, unsigned int epoch) {
  const int lane = threadIdx.x & 31;
  unsigned long long off = 0;
  if (c < OWN_SUM) {
    // (the scanner is still starting: a small launch would wait for it)
    unsigned int sum = 0;
    const uint16_t* table = reinterpret_cast<const uint16_t*>(A.in + HDR);
    for (int i = lane; i < (int)c; i += 32) sum += table[i];
    off = __reduce_add_sync(0xffffffffu, sum);
  } else {
    if (lane == 0) off = wait_offset(A.sy, epoch, c);
    off = __shfl_sync(0xffffffffu, off, 0);
  }
  return off;
}
__device__ __noinline__ unsigned long long open_offset_far(const OpArgs& A, long long c, unsigned int epoch) {
  return open_offset(A, c, epoch);
}

// Second part, once the place at byte `at` (a multiple of 16) of P is free: the
// payload's 16-byte-aligned span with one bulk copy, the ragged tail by the
// lanes.  FAR: the rare wait for an offset is out of line.  The re-encoders hold
// five copies of this, and instruction fetch is their largest stall (128 MiB:
// init_send 152 -> 148 us on nearly all zero bins, init_send_apply 156 -> 152 on
// sinusoids with noise); resi_recv ran 2% slower with it.
template <bool FAR, class Src>
__device__ __forceinline__ void issue_stream(Ctl& sm, int t, const Src& src, uint8_t* P, int at) {
  const int lane = threadIdx.x & 31;
  StageMeta& m = sm.st[t];
  if (m.g >= src.total || m.bad) {
    if (lane == 0) {
      m.csize = 0;
      m.d = 0;
      m.tma_len = 0;
      mbar_arrive(&sm.bar);
      mbar_arrive(&sm.bar);
    }
    return;
  }
  const OpArgs& A = src.args(m.item);
  unsigned long long off = m.off;
  if ((off >> 48) == sm.epoch && (off & LB_INC)) {
    off &= LB_VAL;
  } else {
    off = FAR ? open_offset_far(A, m.c, sm.epoch) : open_offset(A, m.c, sm.epoch);
  }
  const int cs = m.csize;
  __syncwarp();  // (lane 0 rewrites it below)
  const int osize = 4 * m.nw;
  const uint8_t* data = A.in + HDR + 2 * m.chunks;
  const long long data_bytes = A.in_bytes - HDR - 2 * m.chunks;
  const int bad = (cs > osize) || (cs < 2 && cs != osize) || ((long long)off + cs > data_bytes);
  const uintptr_t Aa = reinterpret_cast<uintptr_t>(data + off);
  const uintptr_t a0 = Aa & ~uintptr_t(15);
  uintptr_t a1 = (Aa + (bad ? 0 : cs)) & ~uintptr_t(15);
  if (a1 < a0) a1 = a0;
  // The copy may run into the next payload's bytes: it takes the ragged tail
  // too unless that would read past the stream's valid bytes.
  const uintptr_t a1_up = (Aa + (bad ? 0 : cs) + 15) & ~uintptr_t(15);
  if (!bad && a1_up <= reinterpret_cast<uintptr_t>(A.in + A.in_bytes)) a1 = a1_up;
  const int d = at + (int)(Aa - a0);
  const int tma_len = (int)(a1 - a0);
  if (lane == 0) {
    fence_proxy_async();
    if (tma_len) {
      mbar_expect_tx(&sm.bar, (uint32_t)tma_len);
      bulk_load(P + at, reinterpret_cast<const void*>(a0), (uint32_t)tma_len, &sm.bar);
    } else {
      mbar_arrive(&sm.bar);
    }
    m.bad = bad;
    m.csize = bad ? 0 : cs;
    m.d = d;
    m.tma_len = tma_len;
  }
  if (!bad) {
    const uint8_t* gsrc = data + off;
    const int from = at + tma_len - d;  // payload bytes [from, cs) are copied by the lanes
    for (int i = lane + (from > 0 ? from : 0); i < cs; i += 32) P[d + i] = gsrc[i];
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(&sm.bar);
}

// The client side of a served request, fused into init_send / resi_send
// (cortado_*_send_apply): the words the re-encoder is about to encode (request
// bins, or residuals) are applied to the client's reconstruction directly,
// so the stream just written need not be decoded again.  The results equal
// init_recv / resi_recv of that stream bit for bit:
//   init: iCQ(bin) (d_client_encode.h:230-254); a chunk that the encoder
//         stores uncompressed is rewritten with its bins afterwards
//         (raw_rebuild), as init_recv copies raw chunks out as stored;
//   resi: iCQ(CQ(client, dst) + residual, dst) (d_RESI_4.h:79-94); the
//         residual ints are the same whether the chunk compresses or not.
// A full chunk goes through the stage buffer X, whose rows 32w .. 32w+31
// only warp w touches at this point of the loop (row tid is each thread's
// own): the warp moves its 4 KiB of the client's floats between global and
// those rows 512 contiguous bytes at a time, and each thread works on its own
// row.  The float forms apply when the whole warp allows them (no lossless
// client word, no lossless bin), else the per-word forms, as in the decoders.
// A partial chunk works word by word on the client's floats directly.
template <int OP>
__device__ __noinline__ void client_apply_partial(uint32_t* client, int nw, Quant q, const uint32_t* X) {
  const FastQ fq = make_fastq(q.eb_e);
  for (int w = 32 * threadIdx.x; w < min(32 * (int)threadIdx.x + 32, nw); w++) {
    const uint32_t b = X[swz(w)];
    client[w] = (OP == OP_S2C) ? iq_mixed(b, fq, q) : iq_mixed(cq_mixed(client[w], fq, q) + b, fq, q);
  }
}
template <int OP>
__device__ __forceinline__ void client_apply(const OpArgs& A, long long c, int nw, const uint32_t (&v)[32], Quant q,
                                             uint32_t* X) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const FastQ fq = make_fastq(q.eb_e);
  if (nw == CW) {
    uint4* g4 = reinterpret_cast<uint4*>(A.client) + c * (long long)(CW / 4) + 256 * warp;
    uint4* X4 = reinterpret_cast<uint4*>(X);
    uint4* own = X4 + 8 * tid;
    // lane l's part of the warp's i-th 512 bytes: linear 16-byte unit
    // 256*warp + 32*i + l, i.e. row 32*warp + 4*i + l/8, unit l%8 of that row
    auto unit = [&](int i) -> uint4* {
      const int r = 32 * warp + 4 * i + (lane >> 3);
      return X4 + 8 * r + ((lane & 7) ^ (r & 7));
    };
    __syncwarp();  // the rows' earlier uses by this warp's threads are done
    uint32_t bmax = 0;
    if (OP == OP_S2C) {
#pragma unroll
      for (int k = 0; k < 32; k++) {
        const uint32_t neg = (uint32_t)((int32_t)v[k] >> 31);
        bmax = max(bmax, (v[k] ^ neg) - neg);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++) async_copy16(unit(i), g4 + 32 * i + lane);  // all eight in flight, no registers
      async_wait_all();
      __syncwarp();
      uint32_t amax = 0;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint4 w = own[u ^ (tid & 7)];
        amax = max(amax, max(max(w.x & 0x7fffffffu, w.y & 0x7fffffffu), max(w.z & 0x7fffffffu, w.w & 0x7fffffffu)));
      }
      // destination bins of the client's floats plus the residuals, into the row
      const bool fast_c = !__any_sync(0xffffffffu, amax >= fq.thr_bits);
      __syncwarp();  // the row is read again below, not held in registers beside v
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint4 w = own[u ^ (tid & 7)];
        uint4 b;
        if (fast_c) {
          b = make_uint4(cq_fast(w.x, fq) + v[4 * u], cq_fast(w.y, fq) + v[4 * u + 1], cq_fast(w.z, fq) + v[4 * u + 2],
                         cq_fast(w.w, fq) + v[4 * u + 3]);
        } else {
          b = make_uint4(cq_mixed(w.x, fq, q) + v[4 * u], cq_mixed(w.y, fq, q) + v[4 * u + 1],
                         cq_mixed(w.z, fq, q) + v[4 * u + 2], cq_mixed(w.w, fq, q) + v[4 * u + 3]);
        }
        own[u ^ (tid & 7)] = b;
        const uint32_t b4[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t neg = (uint32_t)((int32_t)b4[j] >> 31);
          bmax = max(bmax, (b4[j] ^ neg) - neg);
        }
      }
    }
    const bool fast_i = __all_sync(0xffffffffu, bmax < 0x800000u);
    if (OP == OP_S2C) {  // the request bins into the row
#pragma unroll
      for (int u = 0; u < 8; u++) own[u ^ (tid & 7)] = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
    }
    __syncwarp();  // the warp's rows hold its bins
    // dequantized on the way out, 512 contiguous bytes at a time
#pragma unroll 2
    for (int i = 0; i < 8; i++) {
      const uint4 b = *unit(i);
      g4[32 * i + lane] = fast_i ? make_uint4(iq_fast(b.x, fq), iq_fast(b.y, fq), iq_fast(b.z, fq), iq_fast(b.w, fq))
                                 : make_uint4(iq_mixed(b.x, fq, q), iq_mixed(b.y, fq, q), iq_mixed(b.z, fq, q),
                                              iq_mixed(b.w, fq, q));
    }
    __syncwarp();  // the rows are read before the encoder reuses the buffer
  } else {
    row_store(X, tid, v);
    client_apply_partial<OP>(reinterpret_cast<uint32_t*>(A.client) + c * (long long)CW, nw, q, X);
  }
}

// The fused forms for a chunk of zeros: request bins of zero are zero as floats;
// residuals of zero move the client's floats to the destination bound's bins.
template <int OP>
__device__ __noinline__ void client_zero(const OpArgs& A, long long c, int nw, Quant q) {
  const FastQ fq = make_fastq(q.eb_e);
  uint32_t* client = reinterpret_cast<uint32_t*>(A.client) + c * (long long)CW;
  auto moved = [&](uint32_t x) -> uint32_t { return (OP == OP_S2C) ? 0u : iq_mixed(cq_mixed(x, fq, q), fq, q); };
  if (nw == CW) {
    uint4* g4 = reinterpret_cast<uint4*>(client) + threadIdx.x;
#pragma unroll 2
    for (int i = 0; i < 8; i++) {
      const uint4 w = (OP == OP_S2C) ? make_uint4(0, 0, 0, 0) : g4[NT * i];
      g4[NT * i] = make_uint4(moved(w.x), moved(w.y), moved(w.z), moved(w.w));
    }
  } else {
    for (int w = threadIdx.x; w < nw; w += NT) client[w] = moved((OP == OP_S2C) ? 0u : client[w]);
  }
}

// Bytes of the re-encoders' R (reencode_loop).
constexpr int ROOM = (2 * BUF_WORDS - CW) * 4;
// Bytes that a payload of n bytes takes at R's high end (any alignment, and
// what the decoder reads past its end), and at its low end (padded).
__host__ __device__ constexpr int room_in(int n) { return ((n + 30) & ~15) + 32; }
__host__ __device__ constexpr int room_out(int n) { return n + (n >> 5) + 32; }
static_assert(room_out(SMALL) + room_in(CS) <= ROOM, "a payload that is not padded is never spilled");
static_assert(room_out(CS) <= 4 * BUF_WORDS, "a payload fits the CTA's place in global memory");

// Rebuilds a raw chunk's requantized words from the planes (X) and spills them.
// Each warp moves its 4 KiB through its own rows of X, 512 contiguous bytes at a
// time.  client (init_send with apply, or null): the chunk's bins replace the
// dequantized words written there, as init_recv emits a raw chunk's bins
// unchanged.  Out of line: only chunks that do not compress take it, and the
// re-encoders' loop is large enough to stall on instruction fetch.
__device__ __noinline__ void raw_rebuild(Ctl& sm, uint32_t* X, int nw, uint32_t* spill, uint32_t* client) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t w[32], before;
  if (nw != CW) widen_planes(X, nw);
  planes_to_words<true>(sm, X, w, before);
  row_store(X, tid, w);
  if (tid == 0) {
    sm.pend[1] = sm.pend[0];
    sm.pend[0].valid = 0;
  }
  __syncwarp();
  const uint4* X4 = reinterpret_cast<const uint4*>(X);
#pragma unroll 2
  for (int i = 0; i < 8; i++) {
    const int r = 32 * warp + 4 * i + (lane >> 3), u = 256 * warp + 32 * i + lane;
    const uint4 x = X4[8 * r + ((lane & 7) ^ (r & 7))];
    __stcg(reinterpret_cast<uint4*>(spill) + u, x);
    if (client) {
      if (4 * u + 4 <= nw) {
        reinterpret_cast<uint4*>(client)[u] = x;
      } else {
        if (4 * u < nw) client[4 * u] = x.x;
        if (4 * u + 1 < nw) client[4 * u + 1] = x.y;
        if (4 * u + 2 < nw) client[4 * u + 2] = x.z;
      }
    }
  }
}

// Writes out a spilled payload (pend[1]); every thread.
template <class Src>
__device__ __noinline__ void flush_spilled(Ctl& sm, const Src src, const uint32_t* spill) {
  const Pend& p = sm.pend[1];
  const OpArgs& Q = src.args(p.item);
  const long long chunks = (Q.n + CS - 1) / CS;
  if (threadIdx.x < 32) {
    const unsigned long long X = lookback_resolve(Q.sy, sm.epoch, p.c, p.csize);
    if (threadIdx.x == 0) sm.payload_off = X;
  }
  __syncthreads();
  const unsigned long long X = sm.payload_off;
  uint8_t* dst = Q.out + HDR + 2 * chunks + X;
  if (p.raw) flush_raw(dst, spill, p.csize);
  else flush_words<false>(dst, spill, p.csize);
  if (threadIdx.x == 0) {
    reinterpret_cast<uint16_t*>(Q.out + HDR)[p.c] = (uint16_t)p.csize;
    if (p.c == chunks - 1) *Q.out_size = HDR + 2 * chunks + (long long)(X + p.csize);
  }
  __syncthreads();
  if (threadIdx.x == 0) sm.pend[1].valid = 0;
}

// Blocking flush of all that is pending, outside the hot path.  Every earlier
// write to R may precede it without a barrier.
template <class Src>
__device__ __noinline__ void flush_now(Ctl& sm, const Src src, uint32_t* R, const uint32_t* spill) {
  __syncthreads();
  resolve_pending(sm, src, sm.pend[0]);
  __syncthreads();
  write_pending<false>(sm, src, sm.pend[0], R, R);
  __syncthreads();
  if (threadIdx.x == 0) sm.pend[0].valid = 0;
  if (sm.pend[1].valid) flush_spilled(sm, src, spill);
}

// Moves the pending payload (padded, at the low end of R) to the CTA's place in
// global memory: the next one does not fit beside it.
// (Waiting for the pending offset instead, to write the payload out, let CTAs
// that had already taken their next chunk wait for one another.  128 MiB,
// init_send: chunks of zeros and random bits mixed 288 -> 203 us, smooth and
// random 332 -> 243, dense 273 -> 247.)
__device__ __noinline__ void spill_now(Ctl& sm, const uint32_t* R, uint32_t* spill) {
  __syncthreads();
  const int n = room_out(sm.pend[0].csize) >> 4;
  const uint4* r = reinterpret_cast<const uint4*>(R);
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += NT) __stcg(reinterpret_cast<uint4*>(spill) + i, r[i]);
  if (threadIdx.x == 0) {
    sm.pend[1] = sm.pend[0];
    sm.pend[0].valid = 0;
  }
  __syncthreads();
}

// Chunks whose words to encode are all zero go without the encode stage: their
// sizes are published at once, and one warp (ZERO_WARP) keeps them until there
// are 32 and then writes their 2-byte payloads, so that no other chunk waits.
// Out of line, and init_send tells such chunks by their stored bins alone: with
// one more live value in its loop it ran 2-5% slower.
constexpr int ZERO_WARP = 2;
template <class Src>
__device__ __noinline__ void zero_flush(Ctl& sm, const Src src) {
  const int lane = threadIdx.x & 31;
  const bool mine = lane < (int)sm.zeros;
  const uint32_t c = mine ? sm.zero_c[lane] : 0u;
  const int item = mine ? sm.zero_item[lane] : 0;
  auto write = [&](uint32_t k, int it, unsigned long long X) {
    const OpArgs& A = src.args(it);
    const long long chunks = (A.n + CS - 1) / CS;
    const uint32_t osize = (uint32_t)min((long long)CS, A.n - k * (long long)CS);
    uint8_t* dst = A.out + HDR + 2 * chunks + X;
    dst[0] = (uint8_t)osize;
    dst[1] = (uint8_t)(osize >> 8);
    reinterpret_cast<uint16_t*>(A.out + HDR)[k] = 2;
    if (k == chunks - 1) *A.out_size = HDR + 2 * chunks + (long long)X + 2;
  };
  bool open = false;  // the offset is not known yet
  if (mine) {
    const unsigned long long f = ld_relaxed(&src.args(item).sy.flags[c]);
    if ((f >> 48) == sm.epoch && (f & LB_INC)) write(c, item, (f & LB_VAL) - 2);
    else open = true;
  }
  for (unsigned int todo = __ballot_sync(0xffffffffu, open); todo; todo &= todo - 1) {
    const int l = __ffs(todo) - 1;
    const uint32_t k = __shfl_sync(0xffffffffu, c, l);
    const int it = __shfl_sync(0xffffffffu, item, l);
    const unsigned long long X = lookback_resolve(src.args(it).sy, sm.epoch, k, 2u);
    if (lane == 0) write(k, it, X);
  }
  __syncwarp();
  if (lane == 0) sm.zeros = 0;
  __syncwarp();
}
// (ZERO_WARP)
template <class Src>
__device__ __noinline__ void zero_chunk(Ctl& sm, const Src src, const StageMeta& m) {
  if ((threadIdx.x & 31) == 0) {
    lookback_publish(src.args(m.item).sy, sm.epoch, m.c, 2u);
    const unsigned int n = sm.zeros;
    sm.zero_c[n] = (uint32_t)m.c;
    sm.zero_item[n] = m.item;
    sm.zeros = n + 1;
  }
  __syncwarp();
  if (sm.zeros == 32) zero_flush(sm, src);
}

// init_send / resi_send (d_s2c_encode_kernel, d_residual_encode_kernel):
// decode the stored chunk, requantize or form the residual, encode.  The first
// 16 KiB of the buffers (Y) hold the BIT_4 planes, first the stored chunk's,
// then the new one's; in between its rows are scratch for the requantization
// and the client's floats.  The 18 KiB behind them (R) hold the previous
// chunk's new payload at the low end, until it is flushed while the new planes
// are read, and the stored payload at the high end; the next one is loaded
// there as soon as this chunk's size is known, or, when the two do not fit,
// after the new payload has been spilled to global memory.  A chunk that does not
// compress stores its requantized words, which are rebuilt from the planes
// (planes_to_words) and always spilled.
// (Decoding in place in one buffer and staging in the other took 11 barriers a
// chunk; this takes 7.  Instruction fetch is then the largest stall beside them,
// hence the loops of planes_to_words, rze_decode and encode_chunk that are not
// unrolled.  128 MiB, init_send and resi_send: sinusoids with noise 252 -> 137 us
// and 256 -> 141, dense data 342 -> 245 and 351 -> 242, nearly all zero bins 159 ->
// 148 and 103 -> 91.)
// APPLY: the fused send-and-apply forms (items with a client's floats); the
// plain forms are compiled without that code.
template <int OP, bool APPLY, class Src>
__device__ __forceinline__ void reencode_loop(Ctl& sm, const Src& src, const Sync& sy) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  init_pack_table();  // (read after the loop's first barrier)
  if (gridDim.x == 1) {
    if (warp == 1) src.scan(sm.epoch);
    __syncthreads();
  }
  uint32_t* Y = stage_buf(sm, 0);
  uint32_t* R = Y + CW;
  uint32_t* spill = sy.spill + (size_t)blockIdx.x * BUF_WORDS;
  const bool feeder = warp == 1;  // (warp 3 packs the densest planes: 1% slower)
  WalkState ws{-1};
  Ahead ah{0, 0};
  auto take = [&]() -> unsigned int { return (feeder && lane == 0) ? next_place(sy) : 0u; };
  auto resolve = [&](int t, unsigned int g) {
    if (feeder) resolve_stream<OP>(sm, t, __shfl_sync(0xffffffffu, g, 0), src, ws, ah);
  };
  auto park = [&](int t) {
    if (feeder) park_stream(sm, t, src, ah);
  };
  auto issue = [&](int t) {  // (feeder)
    issue_stream<true>(sm, t, src, reinterpret_cast<uint8_t*>(R), ROOM - room_in(min(sm.st[t].csize, CS)));
  };
  resolve(0, sm.first);
  park(0);
  if (feeder) issue(0);
  for (int s = 0;; s ^= 1) {  // s: the metadata slot, and the barrier's phase
    if (!mbar_wait(&sm.bar, s, sy.timeout_ns)) latch(sy.status, DST_TIMEOUT);
    const StageMeta& m = sm.st[s];
    if (m.g >= src.total) break;
    const OpArgs& A = src.args(m.item);
    const ChunkKind kind = rze_decode<true>(sm, A.sy, m, R, Y, NoHook{});
    const unsigned int g = take();
    if (Src::batched && m.bad >= 2) {  // unusable stream header (batched): nothing to write
      resolve(s ^ 1, g);
      park(s ^ 1);
      flush_now(sm, src, R, spill);
      if (feeder) issue(s ^ 1);
      continue;
    }
    // The rest of a chunk whose words to encode are all zero.  A payload in R is
    // written out first: CTAs that ran ahead past such chunks made the others wait
    // (sparse fields with 2% of them: init_send 3-5% slower).  A spilled one waits.
    auto zero = [&]() {
      if (warp == ZERO_WARP) zero_chunk(sm, src, m);
      park(s ^ 1);
      if (sm.pend[0].valid) flush_now(sm, src, R, spill);
      if (feeder) issue(s ^ 1);
    };
    if ((OP == OP_S2C || APPLY) && kind == CHUNK_ZERO) {  // request bins and residuals are zero as well
      resolve(s ^ 1, g);
      Quant q1, q2;
      src.quant(m.item, q1, q2);
      if (Src::batched && m.c == 0 && tid == 0) write_header(A.out, m.n, (OP == OP_S2C) ? q1.eb_e : q2.eb_e);
      if (APPLY && A.client) client_zero<OP>(A, m.c, m.nw, q2);
      zero();
      continue;
    }
    uint32_t v[32], before = 0;  // before: the word before this thread's first
    if (kind == CHUNK_ZERO) {
#pragma unroll
      for (int k = 0; k < 32; k++) v[k] = 0;
    } else if (kind == CHUNK_PLANES) {
      planes_to_words<true>(sm, Y, v, before);
    } else {
      row_load(Y, tid, v);
      before = tid ? Y[swz(32 * tid - 1)] : 0u;
      __syncthreads();  // rows are scratch from here on
    }
    uint32_t some = 0;  // plain resi_send: bits set in this thread's residuals
    {
      // stored bins -> floats (iSQ, skipped for chunks stored as floats) ->
      // request bins (CQ, d_s2c.h:132-137) or residuals (d_RESI_4.h:57-76)
      const bool raw = kind == CHUNK_RAW;
      const Quant qs = make_quant(m.eb_e);
      Quant q1, q2;
      src.quant(m.item, q1, q2);
      // Shift form, when every word of the warp allows it: a lossy stored bin
      // a (|a| < 2^23) is the float a * 2^(e_s - 126), so its request bin is
      // a / 2^k1 rounded half away from zero (k1 = e_1 - e_s >= 0), and the
      // residual is a / 2^k2 (rounded) minus that request bin moved to the
      // destination's bins, (a / 2^k1 rounded) << (e_1 - e_2), exact while the
      // latter stays a lossy destination bin (magnitudes below `amax`).
      const int k1 = q1.eb_e - qs.eb_e;
      const int k2 = (OP == OP_RESI) ? q2.eb_e - qs.eb_e : 0;
      const int dd = (OP == OP_RESI) ? q1.eb_e - q2.eb_e : 0;
      // Words the shift form cannot take (lossless stored words, magnitudes
      // at or above amax, every word of a chunk stored raw or of a bound
      // order it does not cover) go through the float path out of line.
      // (amax = 0 when the shift form does not apply: no word qualifies and
      // every word keeps its stored bin for the float path.)
      const bool shift_ok = !raw && k1 >= 0 && k2 >= 0 && dd >= 0;
      const uint32_t amax = !shift_ok ? 0u
                            : (OP == OP_RESI && k2 == 0 && k1 >= 1 && k1 <= 23) ? 0x800000u - (1u << (k1 - 1))
                                                                                 : 0x800000u;
      const uint32_t h1 = shl_clamp(1u, (uint32_t)(k1 - 1)), h2 = shl_clamp(1u, (uint32_t)(k2 - 1));
      auto shifted = [&](uint32_t& w) -> bool {
        const uint32_t neg = (uint32_t)((int32_t)w >> 31);
        const uint32_t a = (w ^ neg) - neg;
        const uint32_t m1 = shr_clamp(a + h1, (uint32_t)k1);
        const uint32_t r = (OP == OP_S2C) ? m1 : shr_clamp(a + h2, (uint32_t)k2) - shl_clamp(m1, (uint32_t)dd);
        const bool ok = a < amax;
        w = ok ? (r ^ neg) - neg : w;
        return ok;
      };
      if (kind != CHUNK_ZERO) {  // (residuals of zero bins are zero)
        uint32_t slow = 0;
#pragma unroll
        for (int k = 0; k < 32; k++) slow |= (shifted(v[k]) ? 0u : 1u) << k;
        const bool slow_before = !shifted(before);
        if (slow | (uint32_t)slow_before) {  // row tid of Y is this thread's own
          row_store(Y, tid, v);
          before = requant_words<OP>(Y, slow, before, slow_before, raw, qs, q1, q2);
          row_load(Y, tid, v);
        }
        if (OP == OP_RESI && !APPLY) {
#pragma unroll
          for (int k = 0; k < 32; k++) some |= v[k];
        }
      }
      if (Src::batched && m.c == 0 && tid == 0) write_header(A.out, m.n, (OP == OP_S2C) ? q1.eb_e : q2.eb_e);
      resolve(s ^ 1, g);
      if (APPLY && A.client) client_apply<OP>(A, m.c, m.nw, v, OP == OP_S2C ? q1 : q2, Y);
    }
    // (the rows of Y are free after the barrier)
    if (OP == OP_S2C || APPLY) {
      __syncthreads();
    } else if (!__syncthreads_or(some != 0)) {
      zero();
      continue;
    }
    Packer pz(0), pk(0);
    const bool raw_out = encode_chunk<false, OP == OP_S2C || APPLY>(
        sm, A.sy, v, before, Y, R, R, m, sm.pend[0], pz, pk,
        [&]() {
          resolve_pending(sm, src, sm.pend[0]);
          park(s ^ 1);
        },
        [&]() { write_pending<false>(sm, src, sm.pend[0], R, R); },
        [&](uint32_t bytes) {
          if (feeder) {
            const int cs = min(sm.st[s ^ 1].csize, CS);
            const bool fits = room_out(min((int)bytes, CS)) + room_in(cs) <= ROOM;
            if (lane == 0) sm.held = (fits ? 0u : 1u) | (sm.pend[1].valid ? 2u : 0u);
            if (fits) issue(s ^ 1);
          }
        });
    __syncthreads();  // the payload's full words are in place
    pz.finish(R);
    pk.finish(R);
    if (raw_out || sm.held) {
      if (sm.held & 2u) flush_spilled(sm, src, spill);
      if (!raw_out && (sm.held & 1u)) spill_now(sm, R, spill);
      if (feeder && (sm.held & 1u)) issue(s ^ 1);  // (R is free: of a raw chunk nothing is staged)
      if (raw_out)
        raw_rebuild(sm, Y, m.nw, spill,
                    OP == OP_S2C && APPLY && A.client ? reinterpret_cast<uint32_t*>(A.client) + m.c * (long long)CW : nullptr);
    }
  }
  if (warp == ZERO_WARP) zero_flush(sm, src);
  flush_now(sm, src, R, spill);
}

// storage decode / init_recv / resi_recv (d_server_decode_kernel,
// d_client_decode_kernel, d_residual_apply_kernel).  Buffer 0 (P) holds the
// payload, buffer 1 (Q) the BIT_4 planes and then the output floats for one
// TMA store.  The next payload is loaded into P as soon as this one has been
// expanded, while the planes are turned back into floats; its size and offset
// are read at the start of the iteration.  resi_recv's client chunk is loaded
// behind the next payload when that is small, else into Q once the planes
// have been read.
template <int OP, class Src>
__device__ __forceinline__ void decode_loop(Ctl& sm, const Src& src, const Sync& sy) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (gridDim.x == 1) {
    if (warp == 1) src.scan(sm.epoch);
    __syncthreads();
  }
  uint32_t* P = stage_buf(sm, 0);
  uint32_t* Q = stage_buf(sm, 1);
  const bool feeder = warp == FEEDER;
  WalkState ws{-1};
  Ahead ah{0, 0};
  long long pending = 0;
  if (feeder) {
    resolve_stream<OP>(sm, 0, sm.first, src, ws, ah);
    if (lane == 0) pending = next_place(sy);
    park_stream(sm, 0, src, ah);
    issue_stream<OP != OP_RAPPLY>(sm, 0, src, reinterpret_cast<uint8_t*>(P), 0);
  }
  uint32_t phase = 0;  // bit 0: payload; bit 1: client chunk
  for (int s = 0;; s ^= 1) {
    if (!mbar_wait(&sm.bar, phase & 1, sy.timeout_ns)) latch(sy.status, DST_TIMEOUT);
    phase ^= 1u;
    const StageMeta& m = sm.st[s];
    if (m.g >= src.total) break;
    if (feeder) {
      // (every other thread is past the previous chunk's last use of this slot)
      const long long gp = __shfl_sync(0xffffffffu, pending, 0);
      if (lane == 0) pending = next_place(sy);
      resolve_stream<OP>(sm, s ^ 1, gp, src, ws, ah);
    }
    const int item = m.item;
    const OpArgs& A = src.args(item);
    const long long c = m.c;
    const int nw = m.nw;
    const bool full = nw == CW;
    if (Src::batched && c == 0 && tid == 0 && m.bad < 2) *A.out_size = m.n;
    auto q_free = [&]() {
      if (tid == TMA_TID) bulk_wait_read();  // the previous chunk's TMA store has read Q
    };
    if (OP != OP_RAPPLY && m.csize == 4 * nw) {
      // Stored uncompressed: copied out as stored, original floats for storage
      // decode (d_server_encode.h:234-249), request bins for init_recv
      // (d_client_encode.h:230-254, the reference's behaviour).  Q is not
      // needed, so the next payload is loaded there at once and the buffers
      // change places: nothing but that load would hide its latency.  The load
      // may complete the barrier's next phase, so the feeder first waits until
      // every warp has seen this one.
      if (feeder) {
        q_free();
        park_stream(sm, s ^ 1, src, ah);
        asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
        issue_stream<OP != OP_RAPPLY>(sm, s ^ 1, src, reinterpret_cast<uint8_t*>(Q), 0);
      } else {
        asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");
      }
      uint32_t* g = reinterpret_cast<uint32_t*>(A.out) + c * (long long)CW;
      const int d = m.d;
#pragma unroll 4
      for (int w = tid; w < nw; w += NT) {
        const int o = d + 4 * w;
        g[w] = __funnelshift_r(P[o >> 2], P[(o >> 2) + 1], 8 * (o & 3));
      }
      uint32_t* const t = P;
      P = Q;
      Q = t;
      __syncthreads();  // the payload and the slot have been read
      continue;
    }
    const ChunkKind kind = rze_decode<OP == OP_RAPPLY>(sm, A.sy, m, P, Q, q_free);
    if (feeder) {
      park_stream(sm, s ^ 1, src, ah);
      issue_stream<OP != OP_RAPPLY>(sm, s ^ 1, src, reinterpret_cast<uint8_t*>(P), 0);
      if (OP == OP_RAPPLY && lane == 0) {
        // When the next payload fills at most the first KiB of P, this chunk's
        // client floats are loaded behind it (1024-byte aligned) now.
        const StageMeta& mn = sm.st[s ^ 1];
        const bool side = full && A.has_map_in && m.bad == 0 && mn.g < src.total && mn.bad == 0 &&
                          mn.tma_len <= 1024 && mn.d + mn.csize <= 1024;
        sm.src_side = side ? 1u : 0u;
        if (side) {
          mbar_expect_tx(&sm.bar_src, CS);
          tma_load_rows(P + 256, src.min(item), (int)(c * 128), &sm.bar_src);
        }
      }
    }
    if (Src::batched && m.bad >= 2) {  // unusable stream header (batched): nothing to write
      __syncthreads();  // every warp has read m.bad: the feeder may take this slot again at once
      continue;
    }
    uint32_t v[32];
    if (kind == CHUNK_ZERO) {
#pragma unroll
      for (int k = 0; k < 32; k++) v[k] = 0;
    } else if (kind == CHUNK_PLANES) {
      uint32_t before;
      planes_to_words<false>(sm, Q, v, before);
    } else if (OP == OP_RAPPLY) {
      row_load(Q, tid, v);
    }
    const Quant q = make_quant(m.eb_e);
    const FastQ fq = make_fastq(m.eb_e);
    if (OP == OP_RAPPLY) {
      // d_iRESI_4 (d_RESI_4.h:79-94): requantize the client's floats to the
      // destination bound, add the residual, dequantize.
      if (kind != CHUNK_PLANES) __syncthreads();  // sm.src_side; Q has been read
      const uint32_t* S = Q;  // where the client's chunk is
      if (full && A.has_map_in) {
        if (sm.src_side) {
          S = P + 256;
        } else if (tid == TMA_TID) {
          fence_proxy_async();
          mbar_expect_tx(&sm.bar_src, CS);
          tma_load_rows(Q, src.min(item), (int)(c * 128), &sm.bar_src);
        }
        if (!mbar_wait(&sm.bar_src, (phase >> 1) & 1, sy.timeout_ns)) latch(sy.status, DST_TIMEOUT);
        phase ^= 2u;
      } else {
        load_plain_rows(Q, A.src, c, nw);
        __syncthreads();
      }
      // The client's words are folded into v in place (client bin + residual).
      // The float forms, chosen per word in a warp that holds lossless client
      // words or bins.
      const uint4* Srow = reinterpret_cast<const uint4*>(S + 32 * tid);
      const int x = tid & 7;
      float amax = 0.0f;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const uint4 w = Srow[u ^ x];
        amax = max3_abs(amax, __uint_as_float(w.x), __uint_as_float(w.y));
        amax = max3_abs(amax, __uint_as_float(w.z), __uint_as_float(w.w));
      }
      if (__all_sync(0xffffffffu, amax < __uint_as_float(fq.thr_bits))) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint4 w = Srow[u ^ x];
          v[4 * u] += cq_fast(w.x, fq);
          v[4 * u + 1] += cq_fast(w.y, fq);
          v[4 * u + 2] += cq_fast(w.z, fq);
          v[4 * u + 3] += cq_fast(w.w, fq);
        }
      } else {
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint4 w = Srow[u ^ x];
          v[4 * u] += cq_mixed(w.x, fq, q);
          v[4 * u + 1] += cq_mixed(w.y, fq, q);
          v[4 * u + 2] += cq_mixed(w.z, fq, q);
          v[4 * u + 3] += cq_mixed(w.w, fq, q);
        }
      }
    }
    // (Zero bins are zero as floats: 128 MiB of zeros 34 -> 32 us.)
    if (OP == OP_RAPPLY || kind == CHUNK_PLANES) {
      // The float form holds for bins up to 2^23 in magnitude (that one is
      // the lossless threshold itself in both forms).
      float f[32], fmax = 0.0f;
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        f[k] = __int2float_rn((int)v[k]);
        f[k + 1] = __int2float_rn((int)v[k + 1]);
        fmax = max3_abs(fmax, f[k], f[k + 1]);
      }
      if (__all_sync(0xffffffffu, fmax <= 8388608.0f)) {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = __float_as_uint(__fmul_rn(f[k], fq.dsc));
      } else {
#pragma unroll
        for (int k = 0; k < 32; k++) v[k] = iq_mixed(v[k], fq, q);
      }
    }
    row_store(Q, tid, v);  // every plane read finished before the decoder's last barrier
    const bool tma_out = full && A.has_map_out;
    if (tma_out) fence_proxy_async();
    __syncthreads();
    if (tma_out) {
      if (tid == TMA_TID) {
        tma_store_rows(src.mout(item), (int)(c * 128), Q);
        bulk_commit();
      }
    } else {
      uint32_t* g = reinterpret_cast<uint32_t*>(A.out) + c * (long long)CW;
      for (int w = tid; w < nw; w += NT) g[w] = Q[swz(w)];
      __syncthreads();
    }
  }
  if (tid == TMA_TID) bulk_wait_read();
}

// ---- the helper CTA of a launch (the first CTA to start, when there are at
// least two): warp 0 runs the lookback resolver (encoders), warp 1 the offset
// scanner (stream inputs).  Being the first to start, it is resident even
// when other kernels share the GPU and not every CTA of the launch fits at
// once, so the CTAs that wait for its offsets cannot wait for a CTA that
// waits for them.  A one-CTA launch scans its offsets itself first.
template <bool RESOLVE, bool SCAN, class Src>
__device__ __forceinline__ void run_helper(Ctl& sm, const Src& src, const Sync& sy) {
  const int warp = threadIdx.x >> 5;
  if (RESOLVE && sy.resolver && warp == 0) resolve_loop(sy, sm.epoch, src.total);
  if (SCAN && warp == 1) src.scan(sm.epoch);
}

// ---- single-stream kernels
__global__ void __launch_bounds__(NT, MINB_STORE) k_store(const __grid_constant__ OpArgs a, const __grid_constant__ CUtensorMap map_in) {
  Ctl& sm = ctl_block();
  Quant q1, q2;
  const unsigned int noa_err = resolve_noa(a, q1, q2);  // every thread, the same result
  const long long chunks = noa_err ? 0 : (a.n + CS - 1) / CS;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (noa_err) {
      latch(a.sy.status, noa_err);  // nothing is written, as the host path writes nothing
    } else {
      write_header(a.out, a.n, q1.eb_e);
      if (chunks == 0) *a.out_size = HDR;
    }
  }
  const SingleSrc src{&a, &map_in, nullptr, chunks, StreamHdr{}, q1, q2};
  if (begin_launch(sm, a.sy)) run_helper<true, false>(sm, src, a.sy);
  else store_loop(sm, src, a.sy);
  finish_launch(sm, a.sy);
}

template <int OP, bool APPLY>
__global__ void __launch_bounds__(NT, MINB_REENC) k_reencode(const __grid_constant__ OpArgs a) {
  Ctl& sm = ctl_block();
  StreamHdr h = read_header(a.in, a.in_bytes);
  const bool hdr_ok = h.ok && h.n == a.n;
  if (!hdr_ok) h.chunks = 0;
  Quant q1, q2;
  const unsigned int noa_err = resolve_noa(a, q1, q2);  // every thread, the same result
  if (noa_err) h.chunks = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (noa_err) {
      latch(a.sy.status, noa_err);  // nothing is written, as the host path writes nothing
    } else {
      if (!hdr_ok) latch(a.sy.status, h.ok ? DST_SIZE_MISMATCH : DST_CORRUPT);
      write_header(a.out, hdr_ok ? h.n : 0, (OP == OP_S2C) ? q1.eb_e : q2.eb_e);
      if (h.chunks == 0) *a.out_size = HDR;
    }
  }
  const SingleSrc src{&a, nullptr, nullptr, h.chunks, h, q1, q2};
  if (begin_launch(sm, a.sy)) run_helper<true, true>(sm, src, a.sy);
  else reencode_loop<OP, APPLY>(sm, src, a.sy);
  finish_launch(sm, a.sy);
}

template <int OP>
__global__ void __launch_bounds__(NT, OP == OP_RAPPLY ? MINB_RAPPLY : MINB_DEC) k_decode(const __grid_constant__ OpArgs a, const __grid_constant__ CUtensorMap map_src,
                                               const __grid_constant__ CUtensorMap map_out) {
  Ctl& sm = ctl_block();
  StreamHdr h = read_header(a.in, a.in_bytes);
  bool hdr_ok = h.ok && h.n <= a.out_cap;
  if (OP == OP_RAPPLY) hdr_ok = hdr_ok && h.n == a.n;
  if (!hdr_ok) h.chunks = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!hdr_ok) latch(a.sy.status, !h.ok ? DST_CORRUPT : (OP == OP_RAPPLY && h.n != a.n) ? DST_SIZE_MISMATCH : DST_CAPACITY);
    *a.out_size = hdr_ok ? h.n : 0;
  }
  const SingleSrc src{&a, &map_src, &map_out, h.chunks, h, a.q1, a.q2};
  if (begin_launch(sm, a.sy)) run_helper<false, true>(sm, src, a.sy);
  else decode_loop<OP>(sm, src, a.sy);
  finish_launch(sm, a.sy);
}

// ---- batched kernels: one persistent launch over many streams.
template <int OP, bool APPLY = false>
__global__ void __launch_bounds__(NT, OP == OP_STORE ? MINB_STORE : (OP == OP_RAPPLY ? MINB_RAPPLY : (OP == OP_S2C || OP == OP_RESI) ? MINB_REENC : MINB_DEC))
k_batch(const BatchItem* __restrict__ items, int n_items, long long total_chunks, const __grid_constant__ Sync sy) {
  Ctl& sm = ctl_block();
  const BatchSrc<OP> src{items, n_items, total_chunks};
  constexpr bool encoder = OP == OP_STORE || OP == OP_S2C || OP == OP_RESI;
  if (begin_launch(sm, sy)) run_helper<encoder, OP != OP_STORE>(sm, src, sy);
  else if (OP == OP_STORE) store_loop(sm, src, sy);
  else if (encoder) reencode_loop<OP, APPLY>(sm, src, sy);
  else decode_loop<OP>(sm, src, sy);
  finish_launch(sm, sy);
}

// ---- store without allocation (cortado_store_encode_noalloc)
// Fixed scratch for callers that cannot allocate device memory: one
// lookback word per chunk for up to CORTADO_NOALLOC_MAX_BYTES of input, then
// the chunk queue, the finished-CTA count, the status word and the epoch
// (32-bit words 0, 1, 2 and 3 of the last 4 entries).  Every GPU that
// loads the library holds this array until the process exits.
constexpr long long NOALLOC_CHUNKS = CORTADO_NOALLOC_MAX_BYTES / CS;
__device__ __align__(256) unsigned long long g_noalloc_scratch[NOALLOC_CHUNKS + 4];

// Same chunk loop as k_store; the last CTA out also reports a device-side
// error as a negative *out_size (there is no context to read it from) and
// clears the status word for the next call (finish_launch).
__global__ void __launch_bounds__(NT, MINB_STORE) k_store_noalloc(const __grid_constant__ OpArgs a,
                                                                  const __grid_constant__ CUtensorMap map_in) {
  Ctl& sm = ctl_block();
  const long long chunks = (a.n + CS - 1) / CS;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    write_header(a.out, a.n, a.q1.eb_e);
    if (chunks == 0) *a.out_size = HDR;
  }
  const SingleSrc src{&a, &map_in, nullptr, chunks, StreamHdr{}, a.q1, a.q2};
  if (begin_launch(sm, a.sy)) run_helper<true, false>(sm, src, a.sy);
  else store_loop(sm, src, a.sy);
  const unsigned int st = finish_launch(sm, a.sy, true);
  if (st) *a.out_size = -(long long)st;
}

// ---- bound verifier (MAXABS_f32, include/verifiers/MAXABS_f32.h:40-72): the
// first index whose reconstruction violates the absolute bound (NaN/Inf must
// match: unequal unless both are NaN), or n if none.
__device__ __forceinline__ bool maxabs_bad(float o, float r, float eb) {
  if (!isfinite(o) || !isfinite(r)) return (r != o) && (!isnan(o) || !isnan(r));
  const float lower = __fsub_rn(o, eb), upper = __fadd_rn(o, eb);
  return (r < lower) || (r > upper) || (fabsf(__fsub_rn(o, r)) > eb);
}

// Bound by DRAM (both arrays once): four pairs of 16-byte loads in flight per
// thread where both arrays allow it (2 x 512 MiB: 277 -> 162 us, 6.6 TB/s; one
// pair of 4-byte loads kept too little in flight), eight pairs of 4-byte loads
// where not (500 us with one pair in this kernel, 273 in one of its own with
// more warps per SM, 192 now).  A thread stops at its first violation, which is
// the lowest of its indices.
__global__ void __launch_bounds__(256) k_verify(const float* __restrict__ orig, const float* __restrict__ recon, long long nw, float eb,
                         unsigned long long* first_bad) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool wide = ((reinterpret_cast<uintptr_t>(orig) | reinterpret_cast<uintptr_t>(recon)) & 15) == 0;
  const long long nv = wide ? nw / 4 : 0;
  const float4* o4 = reinterpret_cast<const float4*>(orig);
  const float4* r4 = reinterpret_cast<const float4*>(recon);
  for (long long i = t; i < nv; i += 4 * stride) {
    float4 o[4], r[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const long long k = min(i + j * stride, nv - 1);  // (the last one again: it changes nothing)
      o[j] = __ldcs(o4 + k);
      r[j] = __ldcs(r4 + k);
    }
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 4; j++)
      bad |= maxabs_bad(o[j].x, r[j].x, eb) | maxabs_bad(o[j].y, r[j].y, eb) | maxabs_bad(o[j].z, r[j].z, eb) |
             maxabs_bad(o[j].w, r[j].w, eb);
    if (bad) {
      for (int j = 0; j < 4; j++) {
        const long long w = 4 * min(i + j * stride, nv - 1);
        for (int b = 0; b < 4; b++) {
          if (maxabs_bad(orig[w + b], recon[w + b], eb)) {
            atomicMin(first_bad, (unsigned long long)(w + b));
            return;
          }
        }
      }
    }
  }
  for (long long i = 4 * nv + t; i < nw; i += 8 * stride) {
    float o[8], r[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const long long k = min(i + j * stride, nw - 1);
      o[j] = orig[k];
      r[j] = recon[k];
    }
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 8; j++) bad |= maxabs_bad(o[j], r[j], eb);
    if (bad) {
#pragma unroll 1
      for (int j = 0; j < 8; j++) {
        const long long k = min(i + j * stride, nw - 1);
        if (maxabs_bad(orig[k], recon[k], eb)) {
          atomicMin(first_bad, (unsigned long long)k);
          return;
        }
      }
    }
  }
}

// ---- NOA range: min/max over the floats, NaNs ignored (fminf/fmaxf skip
// NaN operands).  Each thread keeps four 16-byte loads in flight per pass.
__device__ __forceinline__ unsigned int ordered(float f) {
  const unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// words: ordered-int min and max, and RANGE_DONE words on the count of finished
// blocks, all three reset for the next call by the last block, which hands the
// range over: to the host through mapped pinned memory (a plain store, no copy
// engine, so it is not queued behind bulk copies on other streams), or, when
// host is null, as two floats in device memory for the NOA entry points.
// Bound by DRAM when the field does not fit L2 (512 MiB 91 -> 78 us, 6.9 TB/s
// with what L2 still holds).  A second, one-thread kernel used to hand the range
// over, and every warp, not every block, updated the words: 32 MiB 19.7 -> 8.3
// us, 1 MiB 15.9 -> 10.3 us per queued call.
constexpr int RANGE_DONE = 4;
__global__ void __launch_bounds__(256) k_minmax(const float* x, long long nw, unsigned int* words,
                                                volatile unsigned int* host, float* out) {
  float mn = INFINITY, mx = -INFINITY;
  const long long nv = nw / 4;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  const long long nthr = (long long)gridDim.x * blockDim.x;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long i = t;
  for (; i + 3 * nthr < nv; i += 4 * nthr) {
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = __ldcs(x4 + i + j * nthr);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      mn = fminf(fminf(mn, v[j].x), fminf(v[j].y, fminf(v[j].z, v[j].w)));
      mx = fmaxf(fmaxf(mx, v[j].x), fmaxf(v[j].y, fmaxf(v[j].z, v[j].w)));
    }
  }
  for (; i < nv; i += nthr) {
    const float4 v = x4[i];
    mn = fminf(fminf(mn, v.x), fminf(v.y, fminf(v.z, v.w)));
    mx = fmaxf(fmaxf(mx, v.x), fmaxf(v.y, fmaxf(v.z, v.w)));
  }
  for (long long k = 4 * nv + t; k < nw; k += nthr) {
    mn = fminf(mn, x[k]);
    mx = fmaxf(mx, x[k]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  __shared__ float s_mn[8], s_mx[8];
  if ((threadIdx.x & 31) == 0) {
    s_mn[threadIdx.x >> 5] = mn;
    s_mx[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < 8; w++) {
    mn = fminf(mn, s_mn[w]);
    mx = fmaxf(mx, s_mx[w]);
  }
  atomicMin(&words[0], ordered(mn));
  atomicMax(&words[1], ordered(mx));
  __threadfence();
  if (atomicAdd(&words[RANGE_DONE], 1u) != gridDim.x - 1) return;
  // the last block: every other one's words are in
  __threadfence();
  const unsigned int lo = atomicExch(&words[0], 0xffffffffu), hi = atomicExch(&words[1], 0u);
  words[RANGE_DONE] = 0;
  if (host) {
    host[0] = lo;
    host[1] = hi;
    __threadfence_system();
  } else {
    auto unord = [](unsigned int o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); };
    out[0] = unord(lo);
    out[1] = unord(hi);
  }
}

// Failure-detection self-test: one thread waits, through the decoders' own
// bounded wait, for a payload offset tagged with epoch 0x10000.  Lookback and
// offset words carry a 16-bit epoch, so no launch can ever publish it; the
// wait runs out after the context's timeout, latches DST_TIMEOUT and returns.
__global__ void k_wait_selftest(Sync sy) {
  if (threadIdx.x == 0) (void)wait_offset(sy, 0x10000u, 0);
}

}  // namespace

// ================================================================== host side
// A payload's room per CTA of a re-encoder's largest grid, in device memory.
struct SpillRoom {
  uint32_t* p = nullptr;
  size_t bytes = 0;
  int device = 0;
  unsigned long long context = 0;
};

struct cortado_ctx {
  int device = 0;
  int sms = 0;
  int grid_store = 0, grid_reenc = 0, grid_dec = 0, grid_rapply = 0;
  unsigned long long* flags = nullptr;
  long long flags_cap = 0;
  SpillRoom spill;
  unsigned int* words = nullptr;  // [0] queue, [1] finished, [2] status, [3..4] minmax, [5] epoch, [7] range blocks finished
  int grid_batch[6] = {0, 0, 0, 0, 0, 0};
  int ctas_override[6] = {0, 0, 0, 0, 0, 0};  // per op: resident CTAs per SM (0 = occupancy limit)
  int resolver[6] = {1, 1, 1, 1, 1, 1};        // per op: lookback resolver warp on (encoders)
  // Item tables of the batched launch: a ring of ITEM_SLOTS slots, each with
  // items_cap entries in pinned host staging and in device memory, and an
  // event recorded after the launch that read it.  A call waits only for the
  // launch ITEM_SLOTS calls back, so the host keeps running ahead of the GPU.
  static constexpr int ITEM_SLOTS = 8;
  BatchItem* d_items = nullptr;
  BatchItem* h_items = nullptr;
  int items_cap = 0;
  int items_slot = 0;
  cudaEvent_t items_done[ITEM_SLOTS] = {};
  unsigned int* h_range = nullptr;  // mapped pinned host words: the last NOA range
  unsigned long long timeout_ns = 2000000000ull;
};

namespace {

PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// A float array viewed as rows of 128 bytes, loaded/stored one chunk (128 rows)
// at a time with the 128-byte swizzle.
bool make_rows_map(CUtensorMap* m, const void* base, long long n_bytes) {
  memset(m, 0, sizeof(*m));
  const long long rows = n_bytes / 128;
  if (rows < 128) return false;
  auto fn = tmap_encoder();
  if (!fn) return false;
  cuuint64_t dims[2] = {32, (cuuint64_t)rows};
  cuuint64_t strides[1] = {128};
  cuuint32_t box[2] = {32, 128};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cortado_status from_cuda(cudaError_t e) { return e == cudaSuccess ? CORTADO_OK : (e == cudaErrorMemoryAllocation ? CORTADO_ERR_OOM : CORTADO_ERR_CUDA); }

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int64_t chunks_of(int64_t n) { return (n + CS - 1) / CS; }

cortado_status eb_exponent(float eb, int* e) {
  if (!(eb >= FLT_MIN)) return (eb != eb) ? CORTADO_ERR_EB_TOO_LARGE : CORTADO_ERR_EB_TOO_SMALL;
  uint32_t bits;
  memcpy(&bits, &eb, 4);
  const int be = (int)((bits >> 23) & 0xff);
  if (be + 24 >= 255) return CORTADO_ERR_EB_TOO_LARGE;
  *e = be;
  return CORTADO_OK;
}

cortado_status ensure_flags(cortado_ctx* ctx, int64_t chunks, cudaStream_t st) {
  if (chunks <= ctx->flags_cap) return CORTADO_OK;
  long long cap = 1024;
  while (cap < chunks) cap *= 2;
  if (ctx->flags) {
    cudaStreamSynchronize(st);
    cudaFree(ctx->flags);
    ctx->flags = nullptr;
    ctx->flags_cap = 0;
  }
  // lookback words, then the input payload offsets
  cudaError_t e = cudaMalloc(&ctx->flags, (size_t)cap * 16);
  if (e != cudaSuccess) return from_cuda(e);
  e = cudaMemsetAsync(ctx->flags, 0, (size_t)cap * 16, st);
  if (e != cudaSuccess) return from_cuda(e);
  ctx->flags_cap = cap;
  return CORTADO_OK;
}

// Batch item tables: ITEM_SLOTS tables of at least n_items entries each.
// Growing waits for every launch that reads a table.
cortado_status ensure_items(cortado_ctx* ctx, int n_items) {
  constexpr int SLOTS = cortado_ctx::ITEM_SLOTS;
  if (n_items <= ctx->items_cap) return CORTADO_OK;
  for (cudaEvent_t ev : ctx->items_done) cudaEventSynchronize(ev);  // every table is free
  cudaFree(ctx->d_items);
  cudaFreeHost(ctx->h_items);
  ctx->d_items = nullptr;
  ctx->h_items = nullptr;
  int cap = 64;
  while (cap < n_items) cap *= 2;
  cudaError_t e = cudaMalloc(&ctx->d_items, sizeof(BatchItem) * cap * SLOTS);
  if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_items, sizeof(BatchItem) * cap * SLOTS);
  if (e != cudaSuccess) {
    ctx->items_cap = 0;
    return from_cuda(e);
  }
  ctx->items_cap = cap;
  return CORTADO_OK;
}

Sync next_sync(cortado_ctx* ctx, cudaStream_t, int op = 0) {
  Sync s;
  s.flags = ctx->flags;
  s.offs = ctx->flags + ctx->flags_cap;
  s.flags_cap = ctx->flags_cap;
  s.counter = ctx->words;
  s.status = ctx->words + 2;
  s.epoch = ctx->words + 5;
  s.timeout_ns = ctx->timeout_ns;
  s.resolver = ctx->resolver[op];
  s.spill = ctx->spill.p;
  return s;
}

// A CTA per chunk, and one more for the helper (a one-chunk launch has none), up
// to the persistent grid.  (Without the helper's own CTA, one CTA of a small
// launch worked on two chunks, one after the other.)
int grid_for(int per_sm_grid, int64_t chunks) {
  const long long g = chunks < 2 ? 1 : chunks + 1;
  return (int)(g < per_sm_grid ? g : per_sm_grid);
}

// Grid of an op: the tuned CTAs per SM if set (never above the occupancy
// limit, which `occupancy` holds as a whole-GPU CTA count), else the limit.
int tuned_grid(const cortado_ctx* ctx, int op, int occupancy) {
  const int o = ctx->ctas_override[op];
  if (o <= 0) return occupancy;
  const long long g = (long long)o * ctx->sms;
  return (int)(g < occupancy ? g : occupancy);
}

template <typename K>
int occupancy_grid(K kernel, size_t smem, int sms) {
  int per = 0;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, NT, smem);
  if (per < 1) per = 1;
  return per * sms;
}

constexpr size_t SMEM_STD = smem_bytes(2);  // every encode / decode kernel

cortado_status launch_status(cudaError_t e) { return from_cuda(e == cudaSuccess ? cudaGetLastError() : e); }

}  // namespace

extern "C" {

const char* cortado_status_string(cortado_status s) {
  switch (s) {
    case CORTADO_OK: return "ok";
    case CORTADO_ERR_EB_TOO_SMALL: return "error bound too small";
    case CORTADO_ERR_EB_TOO_LARGE: return "error bound too large";
    case CORTADO_ERR_CORRUPT_STREAM: return "corrupt stream";
    case CORTADO_ERR_SIZE_MISMATCH: return "size mismatch";
    case CORTADO_ERR_TIMEOUT: return "device wait timed out";
    case CORTADO_ERR_OOM: return "out of device memory";
    case CORTADO_ERR_INVALID_ARG: return "invalid argument";
    case CORTADO_ERR_CUDA: return "CUDA error";
    case CORTADO_ERR_ALIGNMENT: return "buffer not 16-byte aligned";
    case CORTADO_ERR_CAPACITY: return "output buffer too small";
    case CORTADO_ERR_SCRATCH_LIMIT: return "input larger than the fixed scratch of the no-allocation entry point";
  }
  return "unknown status";
}

int64_t cortado_max_stream_bytes(int64_t n_bytes) {
  if (n_bytes < 0) return -1;
  const int64_t c = chunks_of(n_bytes);
  return HDR + 2 * c + c * (int64_t)CS;
}

cortado_status cortado_eb_exponent(float eb, int* biased_exponent) {
  int e = 0;
  const cortado_status s = eb_exponent(eb, &e);
  if (s == CORTADO_OK && biased_exponent) *biased_exponent = e;
  return s;
}

// The calling thread's current CUDA context (driver entry point, as for the
// tensor-map encoder), or null when it cannot be queried.
static CUcontext current_context() {
  using Fn = CUresult (*)(CUcontext*);
  static Fn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<Fn>(p);
  });
  CUcontext c = nullptr;
  if (!fn || fn(&c) != CUDA_SUCCESS) return nullptr;
  return c;
}

// The current context's id, never used again in this process, or 0.
static unsigned long long current_context_id() {
  using Fn = CUresult (*)(CUcontext, unsigned long long*);
  static Fn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<Fn>(p);
  });
  const CUcontext c = current_context();
  unsigned long long id = 0;
  return c && fn && fn(c, &id) == CUDA_SUCCESS ? id : 0;
}

// Spill rooms of destroyed contexts, up to four, for the next ones: allocating
// one takes 0.4 to 3 ms, creating a context otherwise 0.1.  A room is used again
// only in the CUDA context that it was allocated in (a device reset or another
// context has another id), and the device has been waited for before it is here.
static SpillRoom g_idle_rooms[4];
static std::mutex g_idle_mu;

static cudaError_t take_room(SpillRoom* room, int device, size_t bytes) {
  const unsigned long long id = current_context_id();
  if (id) {
    std::lock_guard<std::mutex> lock(g_idle_mu);
    for (SpillRoom& r : g_idle_rooms) {
      if (r.p && r.bytes == bytes && r.device == device && r.context == id) {
        *room = r;
        r = SpillRoom{};
        return cudaSuccess;
      }
    }
  }
  *room = SpillRoom{nullptr, bytes, device, id};
  return cudaMalloc(&room->p, bytes);
}
static void give_room(const SpillRoom& room, bool reusable) {
  if (!room.p) return;
  if (reusable && room.context && room.context == current_context_id()) {
    std::lock_guard<std::mutex> lock(g_idle_mu);
    for (SpillRoom& r : g_idle_rooms) {
      if (!r.p) {
        r = room;
        return;
      }
    }
  }
  cudaFree(room.p);
}

cortado_status cortado_create(cortado_ctx** out, int device) {
  if (!out) return CORTADO_ERR_INVALID_ARG;
  *out = nullptr;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return from_cuda(e);
  cortado_ctx* ctx = new cortado_ctx();
  ctx->device = device;
  cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, device);
  e = cudaMalloc(&ctx->words, 64);
  if (e != cudaSuccess) { delete ctx; return from_cuda(e); }
  cudaMemset(ctx->words, 0, 64);
  cudaMemset(ctx->words + 3, 0xff, 4);  // NOA range words: min = all ones, max = 0
  e = cudaHostAlloc((void**)&ctx->h_range, 8, cudaHostAllocMapped);
  if (e != cudaSuccess) { cudaFree(ctx->words); delete ctx; return from_cuda(e); }
  ctx->grid_store = occupancy_grid(k_store, SMEM_STD, ctx->sms);
  ctx->grid_reenc = occupancy_grid(k_reencode<OP_S2C, false>, SMEM_STD, ctx->sms);
  occupancy_grid(k_reencode<OP_RESI, false>, SMEM_STD, ctx->sms);
  occupancy_grid(k_reencode<OP_S2C, true>, SMEM_STD, ctx->sms);  // the fused forms
  occupancy_grid(k_reencode<OP_RESI, true>, SMEM_STD, ctx->sms);
  ctx->grid_dec = occupancy_grid(k_decode<OP_SDEC>, SMEM_STD, ctx->sms);
  occupancy_grid(k_decode<OP_CDEC>, SMEM_STD, ctx->sms);
  ctx->grid_rapply = occupancy_grid(k_decode<OP_RAPPLY>, SMEM_STD, ctx->sms);
  ctx->grid_batch[OP_STORE] = occupancy_grid(k_batch<OP_STORE>, SMEM_STD, ctx->sms);
  ctx->grid_batch[OP_S2C] = occupancy_grid(k_batch<OP_S2C>, SMEM_STD, ctx->sms);
  ctx->grid_batch[OP_RESI] = occupancy_grid(k_batch<OP_RESI>, SMEM_STD, ctx->sms);
  occupancy_grid(k_batch<OP_S2C, true>, SMEM_STD, ctx->sms);  // the fused forms: same shape, attributes set
  occupancy_grid(k_batch<OP_RESI, true>, SMEM_STD, ctx->sms);
  ctx->grid_batch[OP_SDEC] = occupancy_grid(k_batch<OP_SDEC>, SMEM_STD, ctx->sms);
  ctx->grid_batch[OP_CDEC] = occupancy_grid(k_batch<OP_CDEC>, SMEM_STD, ctx->sms);
  ctx->grid_batch[OP_RAPPLY] = occupancy_grid(k_batch<OP_RAPPLY>, SMEM_STD, ctx->sms);
  int ctas = ctx->grid_reenc;
  for (int op : {OP_S2C, OP_RESI}) ctas = ctx->grid_batch[op] > ctas ? ctx->grid_batch[op] : ctas;
  for (cudaEvent_t& ev : ctx->items_done) cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  cortado_status s = from_cuda(take_room(&ctx->spill, device, (size_t)ctas * BUF_WORDS * 4));  // 14.7 MiB on 148 SMs
  if (s == CORTADO_OK) s = ensure_flags(ctx, 1024, 0);
  cudaDeviceSynchronize();
  if (s != CORTADO_OK) { cortado_destroy(ctx); return s; }
  *out = ctx;
  return from_cuda(cudaGetLastError());
}

void cortado_destroy(cortado_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  const bool idle = cudaDeviceSynchronize() == cudaSuccess;
  cudaFree(ctx->flags);
  cudaFree(ctx->words);
  give_room(ctx->spill, idle);
  cudaFree(ctx->d_items);
  cudaFreeHost(ctx->h_items);
  cudaFreeHost(ctx->h_range);
  for (cudaEvent_t ev : ctx->items_done)
    if (ev) cudaEventDestroy(ev);
  delete ctx;
}

cortado_status cortado_set_timeout(cortado_ctx* ctx, uint64_t timeout_ns) {
  if (!ctx || timeout_ns == 0) return CORTADO_ERR_INVALID_ARG;
  ctx->timeout_ns = timeout_ns;
  return CORTADO_OK;
}

cortado_status cortado_reserve(cortado_ctx* ctx, int64_t chunks, int items) {
  if (!ctx || chunks < 0 || items < 0) return CORTADO_ERR_INVALID_ARG;
  cortado_status s = ensure_flags(ctx, chunks, 0);
  if (s) return s;
  if ((s = ensure_items(ctx, items))) return s;
  return from_cuda(cudaStreamSynchronize(0));
}

cortado_status cortado_set_launch_ctas(cortado_ctx* ctx, cortado_op op, int ctas_per_sm) {
  if (!ctx || op < CORTADO_OP_STORE || op > CORTADO_OP_RESI_RECV || ctas_per_sm < 0 || ctas_per_sm > 64)
    return CORTADO_ERR_INVALID_ARG;
  ctx->ctas_override[op] = ctas_per_sm;
  return CORTADO_OK;
}

cortado_status cortado_set_resolver(cortado_ctx* ctx, cortado_op op, int enabled) {
  if (!ctx || op < CORTADO_OP_STORE || op > CORTADO_OP_RESI_RECV) return CORTADO_ERR_INVALID_ARG;
  ctx->resolver[op] = enabled ? 1 : 0;
  return CORTADO_OK;
}

cortado_status cortado_selftest_timeout(cortado_ctx* ctx, cortado_stream_t stream) {
  if (!ctx) return CORTADO_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const Sync sy = next_sync(ctx, st);  // offs holds at least 1024 words from creation
  k_wait_selftest<<<1, 32, 0, st>>>(sy);
  return from_cuda(cudaGetLastError());
}

cortado_status cortado_sync(cortado_ctx* ctx, cortado_stream_t stream) {
  if (!ctx) return CORTADO_ERR_INVALID_ARG;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return from_cuda(e);
  unsigned int st = 0;
  e = cudaMemcpy(&st, ctx->words + 2, 4, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return from_cuda(e);
  if (st) cudaMemset(ctx->words + 2, 0, 4);
  return (cortado_status)st;
}

cortado_status cortado_store_encode(cortado_ctx* ctx, const void* d_in, int64_t n_bytes, float eb_abs, void* d_out,
                                    int64_t out_capacity, int64_t* d_outsize, cortado_stream_t stream) {
  if (!ctx || (!d_in && n_bytes) || !d_out || !d_outsize || n_bytes < 0 || (n_bytes & 3)) return CORTADO_ERR_INVALID_ARG;
  if (!aligned16(d_in) || !aligned16(d_out)) return CORTADO_ERR_ALIGNMENT;
  if (out_capacity < cortado_max_stream_bytes(n_bytes)) return CORTADO_ERR_CAPACITY;
  int e = 0;
  cortado_status s = eb_exponent(eb_abs / 2, &e);  // stored bins use half the bound
  if (s) return s;
  const int64_t chunks = chunks_of(n_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  if ((s = ensure_flags(ctx, chunks, st))) return s;
  OpArgs a{};
  a.in = (const uint8_t*)d_in;
  a.in_bytes = n_bytes;
  a.out = (uint8_t*)d_out;
  a.out_cap = out_capacity;
  a.out_size = (long long*)d_outsize;
  a.n = n_bytes;
  a.q1 = make_quant(e);
  a.sy = next_sync(ctx, st, OP_STORE);
  CUtensorMap map;
  a.has_map_in = make_rows_map(&map, d_in, n_bytes);
  k_store<<<grid_for(tuned_grid(ctx, OP_STORE, ctx->grid_store), chunks), NT, SMEM_STD, st>>>(a, map);
  return launch_status(cudaSuccess);
}

static cortado_status reencode(cortado_ctx* ctx, int op, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                               float eb1, float eb2, void* d_out, int64_t out_capacity, int64_t* d_outsize,
                               cortado_stream_t stream, void* d_client = nullptr, const float* d_minmax = nullptr) {
  if (!ctx || !d_stored || !d_out || !d_outsize || n_bytes < 0 || (n_bytes & 3) || stored_bytes < HDR)
    return CORTADO_ERR_INVALID_ARG;
  if (!aligned16(d_stored) || !aligned16(d_out) || (d_client && !aligned16(d_client))) return CORTADO_ERR_ALIGNMENT;
  if (out_capacity < cortado_max_stream_bytes(n_bytes)) return CORTADO_ERR_CAPACITY;
  int e1 = 1, e2 = 1;
  cortado_status s = CORTADO_OK;
  if (!d_minmax) {  // NOA bounds are checked on the device
    if ((s = eb_exponent(eb1, &e1))) return s;
    if (op == OP_RESI && (s = eb_exponent(eb2, &e2))) return s;
  }
  const int64_t chunks = chunks_of(n_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  if ((s = ensure_flags(ctx, chunks, st))) return s;
  OpArgs a{};
  if (d_minmax) {
    a.noa = d_minmax;
    a.noa_eb1 = eb1;
    a.noa_eb2 = eb2;
    a.noa_mode = (op == OP_S2C) ? 2 : 3;
  }
  a.in = (const uint8_t*)d_stored;
  a.in_bytes = stored_bytes;
  a.out = (uint8_t*)d_out;
  a.out_cap = out_capacity;
  a.out_size = (long long*)d_outsize;
  a.n = n_bytes;
  a.q1 = make_quant(e1);
  a.q2 = make_quant(e2);
  a.client = (uint8_t*)d_client;
  a.sy = next_sync(ctx, st, op);
  const int grid = grid_for(tuned_grid(ctx, op, ctx->grid_reenc), chunks);
  if (op == OP_S2C && d_client) k_reencode<OP_S2C, true><<<grid, NT, SMEM_STD, st>>>(a);
  else if (op == OP_S2C) k_reencode<OP_S2C, false><<<grid, NT, SMEM_STD, st>>>(a);
  else if (d_client) k_reencode<OP_RESI, true><<<grid, NT, SMEM_STD, st>>>(a);
  else k_reencode<OP_RESI, false><<<grid, NT, SMEM_STD, st>>>(a);
  return launch_status(cudaSuccess);
}

cortado_status cortado_init_send(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                 float request_eb_abs, void* d_out, int64_t out_capacity, int64_t* d_outsize,
                                 cortado_stream_t stream) {
  return reencode(ctx, OP_S2C, d_stored, stored_bytes, n_bytes, request_eb_abs, 0.0f, d_out, out_capacity, d_outsize, stream);
}

cortado_status cortado_resi_send(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                 float src_eb_abs, float dst_eb_abs, void* d_out, int64_t out_capacity,
                                 int64_t* d_outsize, cortado_stream_t stream) {
  return reencode(ctx, OP_RESI, d_stored, stored_bytes, n_bytes, src_eb_abs, dst_eb_abs, d_out, out_capacity, d_outsize,
                  stream);
}

cortado_status cortado_init_send_apply(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                       float request_eb_abs, void* d_out, int64_t out_capacity, int64_t* d_outsize,
                                       void* d_client, cortado_stream_t stream) {
  if (!d_client && n_bytes) return CORTADO_ERR_INVALID_ARG;
  return reencode(ctx, OP_S2C, d_stored, stored_bytes, n_bytes, request_eb_abs, 0.0f, d_out, out_capacity, d_outsize,
                  stream, d_client);
}

cortado_status cortado_resi_send_apply(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                       float src_eb_abs, float dst_eb_abs, void* d_out, int64_t out_capacity,
                                       int64_t* d_outsize, void* d_client, cortado_stream_t stream) {
  if (!d_client && n_bytes) return CORTADO_ERR_INVALID_ARG;
  return reencode(ctx, OP_RESI, d_stored, stored_bytes, n_bytes, src_eb_abs, dst_eb_abs, d_out, out_capacity, d_outsize,
                  stream, d_client);
}

cortado_status cortado_noa_range_device(cortado_ctx* ctx, const void* d_in, int64_t n_bytes, float* d_minmax,
                                        cortado_stream_t stream) {
  if (!ctx || !d_in || !d_minmax || n_bytes <= 0 || (n_bytes & 3)) return CORTADO_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const long long nw = n_bytes / 4;
  long long blocks = (nw / 4 + 1023) / 1024;
  if (blocks > 8L * ctx->sms) blocks = 8L * ctx->sms;
  if (blocks < 1) blocks = 1;
  k_minmax<<<(int)blocks, 256, 0, st>>>((const float*)d_in, nw, ctx->words + 3, nullptr, d_minmax);
  return launch_status(cudaSuccess);
}

cortado_status cortado_store_encode_noa(cortado_ctx* ctx, const void* d_in, int64_t n_bytes, const float* d_minmax,
                                        float eb_noa, void* d_out, int64_t out_capacity, int64_t* d_outsize,
                                        cortado_stream_t stream) {
  if (!ctx || (!d_in && n_bytes) || !d_out || !d_outsize || !d_minmax || n_bytes < 0 || (n_bytes & 3))
    return CORTADO_ERR_INVALID_ARG;
  if (!aligned16(d_in) || !aligned16(d_out)) return CORTADO_ERR_ALIGNMENT;
  if (out_capacity < cortado_max_stream_bytes(n_bytes)) return CORTADO_ERR_CAPACITY;
  const int64_t chunks = chunks_of(n_bytes);
  cudaStream_t st = (cudaStream_t)stream;
  cortado_status s = ensure_flags(ctx, chunks, st);
  if (s) return s;
  OpArgs a{};
  a.in = (const uint8_t*)d_in;
  a.in_bytes = n_bytes;
  a.out = (uint8_t*)d_out;
  a.out_cap = out_capacity;
  a.out_size = (long long*)d_outsize;
  a.n = n_bytes;
  a.q1 = make_quant(1);
  a.noa = d_minmax;
  a.noa_eb1 = eb_noa;
  a.noa_mode = 1;
  a.sy = next_sync(ctx, st, OP_STORE);
  CUtensorMap map;
  a.has_map_in = make_rows_map(&map, d_in, n_bytes);
  k_store<<<grid_for(tuned_grid(ctx, OP_STORE, ctx->grid_store), chunks), NT, SMEM_STD, st>>>(a, map);
  return launch_status(cudaSuccess);
}

cortado_status cortado_init_send_noa(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                     const float* d_minmax, float request_eb_noa, void* d_out, int64_t out_capacity,
                                     int64_t* d_outsize, cortado_stream_t stream) {
  if (!d_minmax) return CORTADO_ERR_INVALID_ARG;
  return reencode(ctx, OP_S2C, d_stored, stored_bytes, n_bytes, request_eb_noa, 0.0f, d_out, out_capacity, d_outsize,
                  stream, nullptr, d_minmax);
}

cortado_status cortado_resi_send_noa(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                     const float* d_minmax, float src_eb_noa, float dst_eb_noa, void* d_out,
                                     int64_t out_capacity, int64_t* d_outsize, cortado_stream_t stream) {
  if (!d_minmax) return CORTADO_ERR_INVALID_ARG;
  return reencode(ctx, OP_RESI, d_stored, stored_bytes, n_bytes, src_eb_noa, dst_eb_noa, d_out, out_capacity,
                  d_outsize, stream, nullptr, d_minmax);
}

cortado_status cortado_init_send_apply_noa(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                           const float* d_minmax, float request_eb_noa, void* d_out,
                                           int64_t out_capacity, int64_t* d_outsize, void* d_client,
                                           cortado_stream_t stream) {
  if (!d_minmax || (!d_client && n_bytes)) return CORTADO_ERR_INVALID_ARG;
  return reencode(ctx, OP_S2C, d_stored, stored_bytes, n_bytes, request_eb_noa, 0.0f, d_out, out_capacity, d_outsize,
                  stream, d_client, d_minmax);
}

cortado_status cortado_resi_send_apply_noa(cortado_ctx* ctx, const void* d_stored, int64_t stored_bytes, int64_t n_bytes,
                                           const float* d_minmax, float src_eb_noa, float dst_eb_noa, void* d_out,
                                           int64_t out_capacity, int64_t* d_outsize, void* d_client,
                                           cortado_stream_t stream) {
  if (!d_minmax || (!d_client && n_bytes)) return CORTADO_ERR_INVALID_ARG;
  return reencode(ctx, OP_RESI, d_stored, stored_bytes, n_bytes, src_eb_noa, dst_eb_noa, d_out, out_capacity,
                  d_outsize, stream, d_client, d_minmax);
}

static cortado_status decode(cortado_ctx* ctx, int op, const void* d_stream, int64_t stream_bytes, const void* d_src,
                             int64_t n_bytes, void* d_out, int64_t out_capacity, int64_t* d_outsize,
                             cortado_stream_t stream) {
  if (!ctx || !d_stream || !d_out || !d_outsize || stream_bytes < HDR || out_capacity < 0) return CORTADO_ERR_INVALID_ARG;
  if (!aligned16(d_stream) || !aligned16(d_out) || (d_src && !aligned16(d_src))) return CORTADO_ERR_ALIGNMENT;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t chunk_bound = chunks_of(op == OP_RAPPLY ? n_bytes : out_capacity);
  cortado_status es = ensure_flags(ctx, chunk_bound, st);
  if (es) return es;
  OpArgs a{};
  a.in = (const uint8_t*)d_stream;
  a.in_bytes = stream_bytes;
  a.src = (const uint8_t*)d_src;
  a.out = (uint8_t*)d_out;
  a.out_cap = out_capacity;
  a.out_size = (long long*)d_outsize;
  a.n = n_bytes;
  a.sy = next_sync(ctx, st, op);
  CUtensorMap msrc, mout;
  memset(&msrc, 0, sizeof(msrc));
  // The output map needs the decoded size, which only the stream header holds:
  // cover the whole output capacity (TMA is only used for full chunks, which
  // the kernel checks lie inside the header's size).
  a.has_map_out = make_rows_map(&mout, d_out, op == OP_RAPPLY ? n_bytes : out_capacity);
  if (op == OP_RAPPLY) a.has_map_in = make_rows_map(&msrc, d_src, n_bytes);
  if (op == OP_SDEC) k_decode<OP_SDEC><<<grid_for(tuned_grid(ctx, op, ctx->grid_dec), chunk_bound), NT, SMEM_STD, st>>>(a, msrc, mout);
  else if (op == OP_CDEC) k_decode<OP_CDEC><<<grid_for(tuned_grid(ctx, op, ctx->grid_dec), chunk_bound), NT, SMEM_STD, st>>>(a, msrc, mout);
  else k_decode<OP_RAPPLY><<<grid_for(tuned_grid(ctx, op, ctx->grid_rapply), chunk_bound), NT, SMEM_STD, st>>>(a, msrc, mout);
  return launch_status(cudaSuccess);
}

cortado_status cortado_store_decode(cortado_ctx* ctx, const void* d_stream, int64_t stream_bytes, void* d_out,
                                    int64_t out_capacity, int64_t* d_outsize, cortado_stream_t stream) {
  return decode(ctx, OP_SDEC, d_stream, stream_bytes, nullptr, 0, d_out, out_capacity, d_outsize, stream);
}

cortado_status cortado_init_recv(cortado_ctx* ctx, const void* d_init, int64_t init_bytes, void* d_out,
                                 int64_t out_capacity, int64_t* d_outsize, cortado_stream_t stream) {
  return decode(ctx, OP_CDEC, d_init, init_bytes, nullptr, 0, d_out, out_capacity, d_outsize, stream);
}

cortado_status cortado_resi_recv(cortado_ctx* ctx, const void* d_src, int64_t n_bytes, const void* d_resi,
                                 int64_t resi_bytes, void* d_out, int64_t out_capacity, int64_t* d_outsize,
                                 cortado_stream_t stream) {
  if (!d_src && n_bytes) return CORTADO_ERR_INVALID_ARG;
  if (n_bytes < 0 || (n_bytes & 3) || out_capacity < n_bytes) return n_bytes < 0 || (n_bytes & 3) ? CORTADO_ERR_INVALID_ARG : CORTADO_ERR_CAPACITY;
  return decode(ctx, OP_RAPPLY, d_resi, resi_bytes, d_src, n_bytes, d_out, out_capacity, d_outsize, stream);
}

cortado_status cortado_verify_bound(cortado_ctx* ctx, const void* d_orig, const void* d_recon, int64_t n_bytes,
                                    float eb_abs, unsigned long long* d_first_bad, cortado_stream_t stream) {
  if (!ctx || !d_orig || !d_recon || !d_first_bad || n_bytes < 0 || (n_bytes & 3) || !(eb_abs > 0))
    return CORTADO_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const long long nw = n_bytes / 4;
  cudaError_t e = cudaMemsetAsync(d_first_bad, 0xff, 8, st);
  if (e != cudaSuccess) return from_cuda(e);
  long long blocks = (nw + 255) / 256;
  if (blocks > 8L * ctx->sms) blocks = 8L * ctx->sms;
  if (blocks < 1) blocks = 1;
  k_verify<<<(int)blocks, 256, 0, st>>>((const float*)d_orig, (const float*)d_recon, nw, eb_abs, d_first_bad);
  return launch_status(cudaSuccess);
}

cortado_status cortado_noa_range(cortado_ctx* ctx, const void* d_in, int64_t n_bytes, float* h_min, float* h_max,
                                 cortado_stream_t stream) {
  if (!ctx || !d_in || !h_min || !h_max || n_bytes <= 0 || (n_bytes & 3)) return CORTADO_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const long long nw = n_bytes / 4;
  long long blocks = (nw / 4 + 1023) / 1024;
  if (blocks > 8L * ctx->sms) blocks = 8L * ctx->sms;
  if (blocks < 1) blocks = 1;
  k_minmax<<<(int)blocks, 256, 0, st>>>((const float*)d_in, nw, ctx->words + 3, ctx->h_range, nullptr);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return from_cuda(e);
  const unsigned int r[2] = {((volatile unsigned int*)ctx->h_range)[0], ((volatile unsigned int*)ctx->h_range)[1]};
  auto unord = [](unsigned int o) -> float {
    const unsigned int u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
    float f;
    memcpy(&f, &u, 4);
    return f;
  };
  *h_min = unord(r[0]);
  *h_max = unord(r[1]);
  return CORTADO_OK;
}

cortado_status cortado_batch(cortado_ctx* ctx, cortado_op op, const cortado_item* items, int n_items,
                             cortado_stream_t stream) {
  if (!ctx || !items || n_items <= 0 || op < CORTADO_OP_STORE || op > CORTADO_OP_RESI_SEND_APPLY) return CORTADO_ERR_INVALID_ARG;
  // the fused send-and-apply forms run the re-encoders with the client's floats
  const bool apply = op == CORTADO_OP_INIT_SEND_APPLY || op == CORTADO_OP_RESI_SEND_APPLY;
  if (apply) op = (op == CORTADO_OP_INIT_SEND_APPLY) ? CORTADO_OP_INIT_SEND : CORTADO_OP_RESI_SEND;
  static_assert((int)CORTADO_OP_STORE == OP_STORE && (int)CORTADO_OP_INIT_SEND == OP_S2C &&
                    (int)CORTADO_OP_RESI_SEND == OP_RESI && (int)CORTADO_OP_STORE_DECODE == OP_SDEC &&
                    (int)CORTADO_OP_INIT_RECV == OP_CDEC && (int)CORTADO_OP_RESI_RECV == OP_RAPPLY,
                "op numbering");
  cudaStream_t st = (cudaStream_t)stream;
  // per-item checks, as the single-stream entry points make them
  long long total = 0;
  for (int i = 0; i < n_items; i++) {
    const cortado_item& it = items[i];
    if (!it.d_in || !it.d_out || !it.d_outsize || it.n_bytes <= 0 || (it.n_bytes & 3)) return CORTADO_ERR_INVALID_ARG;
    if (!aligned16(it.d_in) || !aligned16(it.d_out) || (it.d_src && !aligned16(it.d_src))) return CORTADO_ERR_ALIGNMENT;
    int e = 0;
    cortado_status s;
    switch (op) {
      case CORTADO_OP_STORE:
        if (it.in_bytes != it.n_bytes) return CORTADO_ERR_INVALID_ARG;
        if (it.out_capacity < cortado_max_stream_bytes(it.n_bytes)) return CORTADO_ERR_CAPACITY;
        if ((s = eb_exponent(it.eb1 / 2, &e))) return s;
        break;
      case CORTADO_OP_INIT_SEND:
      case CORTADO_OP_RESI_SEND:
        if (it.in_bytes < HDR || (apply && !it.d_src)) return CORTADO_ERR_INVALID_ARG;
        if (it.out_capacity < cortado_max_stream_bytes(it.n_bytes)) return CORTADO_ERR_CAPACITY;
        if ((s = eb_exponent(it.eb1, &e))) return s;
        if (op == CORTADO_OP_RESI_SEND && (s = eb_exponent(it.eb2, &e))) return s;
        break;
      case CORTADO_OP_RESI_RECV:
        if (!it.d_src) return CORTADO_ERR_INVALID_ARG;
        // fall through
      default:
        if (it.in_bytes < HDR) return CORTADO_ERR_INVALID_ARG;
        if (it.out_capacity < it.n_bytes) return CORTADO_ERR_CAPACITY;
        break;
    }
    total += chunks_of(it.n_bytes);
  }
  cortado_status s = ensure_flags(ctx, total, st);
  if (s) return s;
  constexpr int SLOTS = cortado_ctx::ITEM_SLOTS;
  if ((s = ensure_items(ctx, n_items))) return s;
  const int slot = ctx->items_slot;
  ctx->items_slot = (slot + 1) % SLOTS;
  cudaEventSynchronize(ctx->items_done[slot]);  // the launch that last read this slot has ended
  BatchItem* h_tab = ctx->h_items + (size_t)slot * ctx->items_cap;
  BatchItem* d_tab = ctx->d_items + (size_t)slot * ctx->items_cap;
  const Sync sy = next_sync(ctx, st, op);
  long long base = 0;
  for (int i = 0; i < n_items; i++) {
    const cortado_item& it = items[i];
    BatchItem& b = h_tab[i];
    memset(&b, 0, sizeof(b));
    OpArgs& a = b.a;
    a.in = (const uint8_t*)it.d_in;
    a.in_bytes = it.in_bytes;
    a.src = (const uint8_t*)it.d_src;
    a.out = (uint8_t*)it.d_out;
    a.out_cap = it.out_capacity;
    a.out_size = (long long*)it.d_outsize;
    a.n = it.n_bytes;
    int e1 = 1, e2 = 1;
    eb_exponent(op == CORTADO_OP_STORE ? it.eb1 / 2 : it.eb1, &e1);
    eb_exponent(it.eb2, &e2);
    a.q1 = make_quant(e1);
    a.q2 = make_quant(e2);
    a.client = apply ? (uint8_t*)it.d_src : nullptr;
    a.sy = sy;
    a.sy.flags = sy.flags + base;
    a.sy.offs = sy.offs + base;
    if (op == CORTADO_OP_STORE) a.has_map_in = make_rows_map(&b.map_in, it.d_in, it.n_bytes);
    if (op == CORTADO_OP_RESI_RECV) a.has_map_in = make_rows_map(&b.map_in, it.d_src, it.n_bytes);
    if (op == CORTADO_OP_STORE_DECODE || op == CORTADO_OP_INIT_RECV || op == CORTADO_OP_RESI_RECV)
      a.has_map_out = make_rows_map(&b.map_out, it.d_out, it.n_bytes);
    b.chunk_base = base;
    b.chunks = chunks_of(it.n_bytes);
    base += b.chunks;
  }
  cudaError_t e = cudaMemcpyAsync(d_tab, h_tab, sizeof(BatchItem) * n_items, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return from_cuda(e);
  const int grid = grid_for(tuned_grid(ctx, op, ctx->grid_batch[op]), total);
  const size_t smem = (op == CORTADO_OP_RESI_RECV) ? SMEM_STD : SMEM_STD;
  switch (op) {
    case CORTADO_OP_STORE: k_batch<OP_STORE><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy); break;
    case CORTADO_OP_INIT_SEND:
      if (apply) k_batch<OP_S2C, true><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy);
      else k_batch<OP_S2C><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy);
      break;
    case CORTADO_OP_RESI_SEND:
      if (apply) k_batch<OP_RESI, true><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy);
      else k_batch<OP_RESI><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy);
      break;
    case CORTADO_OP_STORE_DECODE: k_batch<OP_SDEC><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy); break;
    case CORTADO_OP_INIT_RECV: k_batch<OP_CDEC><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy); break;
    case CORTADO_OP_RESI_RECV: k_batch<OP_RAPPLY><<<grid, NT, smem, st>>>(d_tab, n_items, total, sy); break;
  }
  cudaEventRecord(ctx->items_done[slot], st);
  return launch_status(cudaSuccess);
}

// Per-device set-up of the no-allocation entry point: the device address of
// g_noalloc_scratch and the persistent grid size, valid for the CUDA context
// that was current when they were looked up (a device reset or a new primary
// context gets a new address, so a change of context repeats the set-up).
struct NoallocDev {
  bool ready = false;
  CUcontext ctx = nullptr;
  unsigned long long* scratch = nullptr;
  int grid = 0;
};

static NoallocDev g_noalloc_dev[64];
static std::mutex g_noalloc_mu;

cortado_status cortado_store_encode_noalloc(const void* d_in, int64_t n_bytes, float eb_abs, void* d_out,
                                            int64_t out_capacity, int64_t* d_outsize, cortado_stream_t stream) {
  if ((!d_in && n_bytes) || !d_out || !d_outsize || n_bytes < 0 || (n_bytes & 3)) return CORTADO_ERR_INVALID_ARG;
  if (n_bytes > CORTADO_NOALLOC_MAX_BYTES) return CORTADO_ERR_SCRATCH_LIMIT;
  if (!aligned16(d_in) || !aligned16(d_out)) return CORTADO_ERR_ALIGNMENT;
  if (out_capacity < cortado_max_stream_bytes(n_bytes)) return CORTADO_ERR_CAPACITY;
  int e = 0;
  cortado_status s = eb_exponent(eb_abs / 2, &e);
  if (s) return s;
  int dev = 0;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) return from_cuda(ce);
  if (dev < 0 || dev >= 64) return CORTADO_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  NoallocDev& d = g_noalloc_dev[dev];
  const CUcontext cur = current_context();
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!d.ready || d.ctx != cur) {
      // device `dev` is current here
      void* p = nullptr;
      ce = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (ce != cudaSuccess) return from_cuda(ce);
      int sms = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      d.grid = occupancy_grid(k_store_noalloc, SMEM_STD, sms);
      d.scratch = (unsigned long long*)p;
      d.ctx = cur;
      d.ready = true;
    }
  }
  OpArgs a{};
  a.in = (const uint8_t*)d_in;
  a.in_bytes = n_bytes;
  a.out = (uint8_t*)d_out;
  a.out_cap = out_capacity;
  a.out_size = (long long*)d_outsize;
  a.n = n_bytes;
  a.q1 = make_quant(e);
  a.sy.flags = d.scratch;
  a.sy.offs = nullptr;
  a.sy.flags_cap = NOALLOC_CHUNKS;
  a.sy.counter = reinterpret_cast<unsigned int*>(d.scratch + NOALLOC_CHUNKS);
  a.sy.status = a.sy.counter + 2;
  a.sy.epoch = a.sy.counter + 3;
  a.sy.timeout_ns = 2000000000ull;
  a.sy.resolver = 1;
  CUtensorMap map;
  a.has_map_in = make_rows_map(&map, d_in, n_bytes);
  k_store_noalloc<<<grid_for(d.grid, chunks_of(n_bytes)), NT, SMEM_STD, st>>>(a, map);
  return launch_status(cudaSuccess);
}

}  // extern "C"

