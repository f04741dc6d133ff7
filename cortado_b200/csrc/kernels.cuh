// Arguments, shared-memory layout and small pieces that the kernels' per-chunk
// stages (decode.cuh, encode.cuh) share.  Reference counterparts:
//   store encode   include/d_server_encode.h:51-143
//   storage decode include/d_server_encode.h:174-260
//   init_send      include/d_s2c.h:51-200
//   init_recv      include/d_client_encode.h:173-259
//   resi_send      include/d_residual_encode.h:51-201
//   resi_recv      include/d_residual_encode.h:238-347
// Differences in mechanism (not in output bytes): output offsets from a
// bounded, epoch-tagged decoupled lookback, resolved one chunk later
// (encoders), and input offsets from a prefix sum of the size table computed
// once per launch (decoders, re-encoders); one 128-thread CTA per chunk with
// the data held in registers; TMA for float chunks and compressed payloads;
// errors latched in a status word instead of printf + __trap.
#pragma once
#include "device.cuh"

namespace cortado {

enum Op : int { OP_STORE = 0, OP_S2C = 1, OP_RESI = 2, OP_SDEC = 3, OP_CDEC = 4, OP_RAPPLY = 5 };

struct OpArgs {
  const uint8_t* in;        // store: floats; others: input stream
  long long in_bytes;       // store: N; others: valid bytes of the input stream
  const uint8_t* src;       // resi_recv: client floats
  uint8_t* out;             // output stream or floats
  long long out_cap;
  long long* out_size;      // device
  long long n;              // original bytes (host-known for encoders; 0 = read header)
  Quant q1, q2;             // store: server; init_send: request; resi_send: src, dst
  Sync sy;
  int has_map_in, has_map_out;
  uint8_t* client;          // init_send / resi_send with apply: the client's reconstruction (floats), or null
  // NOA bounds resolved on the device (cortado_*_noa): q1/q2 come from
  // noa_eb1/noa_eb2 times the range max - min of noa[0..1] (device floats)
  const float* noa;
  float noa_eb1, noa_eb2;
  int noa_mode;             // 0: q1/q2 as given; 1: store (half of eb1); 2: init (eb1); 3: residual (eb1, eb2)
};

// The NOA bounds of the drivers (src/cortado_store.cu:222-227,
// src/cortado_init.cu:294-296, src/cortado_resi.cu:329-332), evaluated on the
// device: eb_abs = float(max - min) * eb, each step rounded once, the store's
// bins at eb_abs / 2, then the checks and biased exponent of the host-side
// eb_exponent.  Returns 0 or the status to latch.
__device__ __forceinline__ unsigned int noa_exponent(float eb, int* e) {
  if (!(eb >= 1.17549435e-38f)) return (eb != eb) ? DST_EB_TOO_LARGE : DST_EB_TOO_SMALL;  // FLT_MIN
  const int be = (int)((__float_as_uint(eb) >> 23) & 0xffu);
  if (be + 24 >= 255) return DST_EB_TOO_LARGE;
  *e = be;
  return 0;
}
__device__ __forceinline__ unsigned int resolve_noa(const OpArgs& a, Quant& q1, Quant& q2) {
  q1 = a.q1;
  q2 = a.q2;
  if (!a.noa_mode) return 0;
  const float range = __fsub_rn(a.noa[1], a.noa[0]);
  float eb1 = __fmul_rn(range, a.noa_eb1);
  if (a.noa_mode == 1) eb1 = __fdiv_rn(eb1, 2.0f);  // stored bins use half the bound
  int e1 = 1, e2 = 1;
  unsigned int st = noa_exponent(eb1, &e1);
  if (!st && a.noa_mode == 3) st = noa_exponent(__fmul_rn(range, a.noa_eb2), &e2);
  if (st) return st;
  q1 = make_quant(e1);
  if (a.noa_mode == 3) q2 = make_quant(e2);
  return 0;
}

// ---------------------------------------------------------------- shared memory
// A CTA owns a 1 KiB control block followed by two chunk buffers of
// BUF_WORDS words (16 KiB + slack, a multiple of 1024 bytes so that every
// buffer keeps the 1024-byte alignment TMA's 128B swizzle needs).  How the
// loops use them is described at each loop (cortado.cu).
constexpr int BUF_WORDS = 4352;
constexpr int CTL_BYTES = 1024;

// What the prefetch of one queue entry found (written by the prefetching warp,
// read by all threads in the iteration that processes it).
struct StageMeta {
  long long g;              // queue index (>= the queue length: no chunk)
  long long c;              // chunk within its stream
  long long n;              // stream's original bytes
  long long chunks;         // stream's chunks
  unsigned long long off;   // decoders: the scanner's word (payload offset in the stream's data section)
  int item;                 // batched launches: the stream
  int nw;                   // words in the chunk
  int tma;                  // store: the floats come by TMA (else the CTA copies them)
  int bad;                  // 1: corrupt size entry; 2: unusable stream header
  int csize;                // decoders: payload bytes
  int d;                    // decoders: payload's byte offset in its buffer
  int tma_len;              // decoders: bytes brought by the bulk copy
  int eb_e;                 // decoders: the stream's exponent
};

// The chunk whose payload waits in a staging buffer for its output offset
// (written by thread 0 in encode_chunk, flushed one iteration later).
struct Pend {
  long long c;
  int item;
  int nw;
  int csize;
  int raw;                  // stored uncompressed
  int small;                // staged without padding
  int valid;
};

struct __align__(16) Ctl {
  uint16_t l2[NT];          // level-2 bitmap (2 bytes per segment thread)
  uint32_t scan_a[4], scan_b[4], scan_c[4];
  uint64_t bar;             // a chunk's loads
  uint64_t bar_src;         // resi_recv: the client chunk
  StageMeta st[2];
  Pend pend[2];             // encoders: the chunks whose payloads wait to be flushed (re-encoders: [1] a spilled one)
  unsigned long long payload_off;
  unsigned int epoch, is_last;
  unsigned int first;       // the CTA's first place in the queue (all ones: the helper)
  unsigned int held;        // re-encoders: bit 0: the next payload waits for room; bit 1: pend[1] is to be flushed
  unsigned int src_side;    // resi_recv: this chunk's client floats are behind the next payload
  unsigned int zeros;       // re-encoders: chunks of zeros whose 2-byte payloads wait for their offsets
  uint32_t zero_c[32];      //   (chunk and item of each; one warp's alone)
  int zero_item[32];
};
static_assert(sizeof(Ctl) <= CTL_BYTES, "control block");

__host__ __device__ constexpr size_t smem_bytes(int nbuf) { return CTL_BYTES + (size_t)nbuf * BUF_WORDS * 4 + 1024; }

__device__ __forceinline__ uint32_t* stage_buf(Ctl& sm, int k) {
  return reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(&sm) + CTL_BYTES + k * (BUF_WORDS * 4));
}

struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};

// Writes `csize` payload bytes to global memory at dst (any alignment) with
// 16-byte stores for the aligned interior.  word(q) returns payload word q
// (bytes 4q..4q+3, little-endian).  UNROLL: blocks in flight per thread.
template <int UNROLL = 1, typename WordFn>
__device__ __forceinline__ void store_payload(uint8_t* dst, int csize, WordFn word) {
  const int tid = threadIdx.x;
  const uintptr_t A = reinterpret_cast<uintptr_t>(dst);
  const uintptr_t a0 = (A + 15) & ~uintptr_t(15);
  const uintptr_t a1 = (A + csize) & ~uintptr_t(15);
  auto byte_at = [&](int i) -> uint8_t { return (uint8_t)(word(i >> 2) >> (8 * (i & 3))); };
  if (a1 > a0) {
    const int head = (int)(a0 - A);
    const int nblk = (int)((a1 - a0) >> 4);
    const int r = head & 3;
#pragma unroll(UNROLL)
    for (int b = tid; b < nblk; b += NT) {
      const int o = head + 16 * b;
      const int q = o >> 2;
      uint32_t w0 = word(q), w1 = word(q + 1), w2 = word(q + 2), w3 = word(q + 3);
      if (r) {
        const uint32_t w4 = word(q + 4);
        w0 = __funnelshift_r(w0, w1, 8 * r);
        w1 = __funnelshift_r(w1, w2, 8 * r);
        w2 = __funnelshift_r(w2, w3, 8 * r);
        w3 = __funnelshift_r(w3, w4, 8 * r);
      }
      *reinterpret_cast<uint4*>(a0 + 16 * (uintptr_t)b) = make_uint4(w0, w1, w2, w3);
    }
    if (tid < head) dst[tid] = byte_at(tid);
    const int tail = (int)(A + csize - a1);
    if (tid < tail) dst[(a1 - A) + tid] = byte_at((int)(a1 - A) + tid);
  } else {
    for (int i = tid; i < csize; i += NT) dst[i] = byte_at(i);
  }
}

// Physical plane-buffer word offsets of linear word s*128 + tid for even and
// odd s (full chunk): the swizzle term depends on s only through its parity,
// so the 32 plane words of a thread sit at base + 128*s + (s odd ? o : e).
__device__ __forceinline__ void plane_offsets(int tid, uint32_t& e, uint32_t& o) {
  const uint32_t lane = tid & 31, warp = tid >> 5;
  e = 32 * warp + ((((lane >> 2) & 7u) ^ warp) << 2) + (lane & 3);
  o = 32 * warp + ((((lane >> 2) & 7u) ^ (warp + 4)) << 2) + (lane & 3);
}

// The partial last chunk of a stream (nw < 4096 words, G whole groups and a
// remainder that BIT_4 copies untransposed) runs through the full chunks' code:
// these two move its BIT_4 output (plane s at words s*G .. s*G+G-1, then the
// remainder) to and from the full chunk's place in a plane buffer (plane s at
// words 128*s ..), padded with zeros.  Eight planes move per step, in the order
// in which no step writes over a later one's source; warp 0 transposes the
// remainder with one vote per plane or word.  Out of line and short: small
// launches mostly wait for instructions to be fetched, and a partial chunk ends
// them (a second copy of the stages for partial chunks took 4 us more).
// Called by every thread; ends with a barrier, expects one before.
__device__ __noinline__ void widen_planes(uint32_t* Y, int nw) {
  const int tid = threadIdx.x, lane = tid & 31, G = nw >> 5, rem = nw & 31;
  uint32_t z = (tid < rem) ? Y[swz(32 * G + tid)] : 0u, mine = 0;
  if (tid < 32) {
    for (int s = 0; s < 32; s++) {
      const uint32_t p = __brev(__ballot_sync(0xffffffffu, (z >> (31 - s)) & 1u));
      if (lane == s) mine = p;  // plane s of the remainder
    }
  }
#pragma unroll 1
  for (int s0 = 24; s0 >= 0; s0 -= 8) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = tid < G ? Y[swz((s0 + i) * G + tid)] : 0u;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++) Y[swz(128 * (s0 + i) + tid)] = v[i];
    __syncthreads();
  }
  if (tid < 32) Y[swz(128 * tid + G)] = mine;
  __syncthreads();
}
__device__ __noinline__ void compact_planes(uint32_t* Y, int nw) {
  const int tid = threadIdx.x, lane = tid & 31, G = nw >> 5, rem = nw & 31;
  uint32_t p = tid < 32 ? Y[swz(128 * tid + G)] : 0u, mine = 0;
  if (tid < 32) {
    for (int k = 0; k < rem; k++) {
      const uint32_t z = __brev(__ballot_sync(0xffffffffu, (p >> (31 - k)) & 1u));
      if (lane == k) mine = z;  // word k of the remainder
    }
  }
#pragma unroll 1
  for (int s0 = 0; s0 < 32; s0 += 8) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = Y[swz(128 * (s0 + i) + tid)];
    __syncthreads();
    if (tid < G) {
#pragma unroll
      for (int i = 0; i < 8; i++) Y[swz((s0 + i) * G + tid)] = v[i];
    }
    __syncthreads();
  }
  for (int w = 32 * G + tid; w < CW; w += NT) Y[swz(w)] = w < nw ? mine : 0u;  // (tid < rem in warp 0 holds word tid)
  __syncthreads();
}

// Inverse of DIFFMS + BIT_4 for a chunk whose BIT_4 output sits in the
// swizzled plane buffer: gathers the plane words of group g = threadIdx.x,
// transposes them back, undoes the zig-zag and the differences (in-thread
// prefix sum plus a block scan of the group totals), and returns the group's
// words in v[32] and the word before them in `before` (0 for the first group).
// The planes are taken a half at a time, as encode_chunk writes them.
// (Words behind a partial chunk's end repeat its last one.)  Ends with a
// barrier (the scan's), after which the plane buffer may be reused.  SHORT:
// loops are not unrolled (the re-encoders, whose code is long).
template <bool SHORT>
__device__ __forceinline__ void planes_to_words(Ctl& sm, const uint32_t* plane, uint32_t (&v)[32], uint32_t& before) {
  const int tid = threadIdx.x;
  // ---- undo BIT_4 (d_iBIT_4): gather plane words of group g, transpose.
  uint32_t pe, po;
  plane_offsets(tid, pe, po);
  uint32_t h[16], p[16];  // planes 0..15 and 16..31, transposed
#pragma unroll
  for (int s = 0; s < 16; s++) p[s] = 0;
  bool wide = false, live = false;  // planes 0..15, 16..31 hold something
#pragma unroll(SHORT ? 1 : 2)
  for (int half = 0; half < 2; half++) {
    uint32_t any = 0;
#pragma unroll
    for (int s = 0; s < 16; s++) {
      h[s] = p[s];
      p[s] = plane[2048 * half + 128 * s + ((s & 1) ? po : pe)];
      any |= p[s];
    }
    wide = live;
    if (__any_sync(0xffffffffu, any != 0)) {
      transpose_blocks(p);
      live = true;
    }
  }
  // ---- undo DIFFMS (d_iDIFFMS, d_DIFFMS.h:69-102): un-zig-zag (z to z / 2, or
  // its complement when z is odd), prefix sum.
  uint32_t acc = 0;
  if (wide) {
#pragma unroll
    for (int k = 0; k < 16; k++) {
      v[k] = __byte_perm(p[k], h[k], 0x7632);
      v[k + 16] = __byte_perm(p[k], h[k], 0x5410);
    }
#pragma unroll
    for (int k = 0; k < 32; k++) {
      const uint32_t u = v[k] >> 1;
      acc += u ^ (2u * u - v[k]);  // 2u - z is 0 or -1: z's low bit
      v[k] = acc;
    }
  } else {
    // 16-bit words, two to a register: differences of 16 bits, summed by two-way
    // dot products with (1, 0) and (0, 1) (256 MiB: init_recv 134 -> 128 us,
    // init_send 281 -> 268 us on sinusoids with noise)
#pragma unroll
    for (int k = 0; k < 16; k++) p[k] = ((p[k] >> 1) & 0x7fff7fffu) ^ ((p[k] & 0x00010001u) * 0xffffu);
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = acc = (uint32_t)__dp2a_lo((int)p[k], 0x0100, (int)acc);
#pragma unroll
    for (int k = 0; k < 16; k++) v[k + 16] = acc = (uint32_t)__dp2a_lo((int)p[k], 0x0001, (int)acc);
  }
  uint32_t total;
  const uint32_t carry = block_scan_excl(acc, sm.scan_c, total);  // (its barrier: every plane read is done)
#pragma unroll
  for (int k = 0; k < 32; k++) v[k] += carry;
  before = carry;
}

}  // namespace cortado
