// The encoders' per-chunk stage: DIFFMS, BIT_4 and RZE_1 of one 16 KiB chunk
// in a 128-thread CTA, 32 words per thread (the layouts of device.cuh), the
// raw fallback, and the staging of the payload until its output offset is
// known.
//
// What bounds it: the integer pipe (48-51% busy) and the barriers between a
// chunk's phases (half the stalls), not DRAM.  Hence:
//   * words below 2^16 (nearly all differences of neighbours) are transposed in
//     16 registers instead of 32;
//   * the zero-byte bitmap comes from byte dot products (36 instructions for
//     eight words; 56 with shifts and multiplies, and the store took 5% longer);
//   * the payload is packed from registers into full words (15 instructions a
//     word) instead of byte by byte, over the planes, whose buffer no thread
//     reads any more; the other buffer is free for the next chunk's input;
//   * only warp 0 derives the small bitmap levels, unless the chunk is close
//     to being stored raw;
//   * few bytes are written one by one, behind the planes: the packing's fixed
//     cost is higher than theirs.
// Store of 128 MiB: 151 -> 80 us (sinusoids with noise, 30% of the size), 174 ->
// 114 (dense, 82%), 94 -> 85 (nearly all zero bins).
#pragma once
#include "decode.cuh"

namespace cortado {

// ---------------------------------------------------------------- staging
// Payload word w of a staged chunk sits at word w + w / 32: threads write runs
// of words that start about 32 words apart, and the padding spreads those over
// the banks (as it does the flush's reads, four words apart per lane).
// A small payload is not padded.
__device__ __forceinline__ uint32_t staged(uint32_t w) { return w + (w >> 5); }
__device__ __forceinline__ uint8_t* staged_byte(uint32_t* st, uint32_t p, bool small) {
  return reinterpret_cast<uint8_t*>(st) + (small ? p : p + ((p >> 7) << 2));
}

// Largest payload staged behind the planes, where it needs no padding (240 words of the 256 there, with
// the words that a flush reads past the end).
constexpr uint32_t SMALL = 960;

// Compaction selectors: entry m packs the bytes of a word that the nibble m
// selects to the low end (byte-permute selector, zero above) and holds eight
// times their number in its upper half.
__device__ __forceinline__ uint32_t* pack_table() {
  __shared__ __align__(64) uint32_t table[16];
  return table;
}
__device__ __forceinline__ void init_pack_table() {
  if (threadIdx.x < 16) {
    const uint32_t m = threadIdx.x;
    uint32_t sel = 0, n = 0;
    for (uint32_t b = 0; b < 4; b++)
      if ((m >> b) & 1) sel |= b << (4 * n++);
    for (uint32_t i = n; i < 4; i++) sel |= 4u << (4 * i);
    pack_table()[m] = sel | (8 * n) << 16;
  }
}
// Entry of nibble i of M.
__device__ __forceinline__ uint32_t pack_entry(uint32_t M, int i) {
  const uint32_t off = (i ? M >> (4 * i - 2) : M << 2) & 60u;
  return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(pack_table()) + off);
}

// A thread's run of payload bytes, written a full word at a time.  Of the word
// that a run starts in, the bytes before it (earlier threads' last ones) are
// stored as zeros; of the word that it ends in, a thread keeps its bytes (acc)
// and adds them in finish(), after the barrier that follows every thread's
// put()s.  t: the run's end so far, in bits.
struct Packer {
  uint32_t acc, t;
  __device__ __forceinline__ explicit Packer(uint32_t p) : acc(0), t(8 * p) {}
  __device__ __forceinline__ void put(uint32_t* st, uint32_t x, uint32_t entry) {
    const uint32_t y = prmt(x, 0u, entry);
    const uint32_t lo = acc | __funnelshift_l(0u, y, t), hi = __funnelshift_l(y, 0u, t);  // (the shifts use t % 32)
    const uint32_t w = t >> 5;
    const uint32_t n = t + (entry >> 16);
    const bool full = (n ^ t) & 32u;
    if (full) st[staged(w)] = lo;
    acc = full ? hi : lo;
    t = n;
  }
  __device__ __forceinline__ void finish(uint32_t* st) const {
    if (acc) atomicOr(st + staged(t >> 5), acc);
  }
};

// ============================================================== encode stage
// Input: v[32] = the pre-DIFFMS words of group g = threadIdx.x (quantized bins
// or residuals; anything at or beyond m.nw) and, for lane 0, the word before
// them (prev0, 0 for thread 0).  Y is free on entry; it becomes the plane
// buffer (d_DIFFMS_4 -> d_BIT_4 -> d_RZE_1, raw fallback).  The payload goes,
// padded (staged()), to `st`, which may be Y itself and is not written before
// the planes have been read, or unpadded to `st_small` (not Y) when it has at
// most SMALL bytes, and stays there until flush_staged writes it out.  The
// chunk's size is published for the lookback and the chunk recorded in `pend`.
// Returns whether the chunk is stored raw; then nothing is staged and the
// planes are still in Y.  The caller holds a barrier after this, then every
// thread finishes its runs pz and pk.
// Three hooks run on every thread: planes_written() before the barrier after
// which the planes are read, planes_ready() after it, and planes_read(n) after
// the next one, with a bound n of the payload's bytes.
// Full groups are transposed one half of the planes at a time: words k and k + 16
// share a register (their high halves for planes 0..15, their low halves for
// planes 16..31), and the stages run on 16 registers.  The pass for planes that
// are zero in the whole warp is left out, and both passes are the same code.
// KEEP: the plane words stay in registers (st is Y); else they are read again for
// the packing, eight at a time in a loop, which keeps the re-encoders' code short.  ZEROS: the words may all be zero (else the caller
// has seen to such chunks).
template <bool KEEP, bool ZEROS, typename Written, typename Ready, typename Read>
__device__ __forceinline__ bool encode_chunk(Ctl& sm, const Sync& sy, uint32_t (&v)[32], uint32_t prev0, uint32_t* Y,
                                             uint32_t* st, uint32_t* st_small, const StageMeta& m, Pend& pend, Packer& pz, Packer& pk,
                                             Written planes_written, Ready planes_ready, Read planes_read) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = m.nw;
  const int osize = nw * 4;
  pz.acc = pk.acc = 0;

  // DIFFMS (d_DIFFMS.h:44-66): word minus its predecessor, then zig-zag.
  uint32_t prev = __shfl_up_sync(0xffffffffu, v[31], 1);
  if (lane == 0) prev = prev0;
  uint32_t any = 0;
#pragma unroll
  for (int k = 0; k < 32; k++) {
    const uint32_t cur = v[k];
    const uint32_t d = cur - prev;
    prev = cur;
    v[k] = (d << 1) ^ (uint32_t)((int32_t)d >> 31);
    any |= v[k];
  }
  // BIT_4: thread g's words are transposed into the planes (plane s at linear
  // words 128 s ..; the warp's part of it is row 4 s + warp of Y).
  const uint32_t bits = __reduce_or_sync(0xffffffffu, any);
  uint32_t pe, po;
  plane_offsets(tid, pe, po);
  int half = 0;
  if (bits < 0x10000u) {  // planes 0..15 are zero: lanes 2s and 2s + 1 clear row s
    half = 1;
    uint4* r = reinterpret_cast<uint4*>(Y + 32 * (4 * (lane >> 1) + warp));
#pragma unroll
    for (int u = 0; u < 4; u++) r[((lane & 1) << 2 | u) ^ ((lane >> 1) & 7)] = make_uint4(0, 0, 0, 0);
  }
#pragma unroll 1
  for (; half < 2; half++) {
    uint32_t p[16];
#pragma unroll
    for (int k = 0; k < 16; k++) p[k] = prmt(v[k], v[k + 16], half ? 0x1054u : 0x3276u);
    if (bits) transpose_blocks(p);
#pragma unroll
    for (int s = 0; s < 16; s++) Y[2048 * half + 128 * s + ((s & 1) ? po : pe)] = p[s];
  }
  if (nw != CW) {
    __syncthreads();
    compact_planes(Y, nw);
  }
  planes_written();
  bool any_nz = true;
  if (ZEROS) any_nz = __syncthreads_or(any != 0);
  else __syncthreads();
  planes_ready();
  if (!any_nz) {
    // No difference at all: zero elimination leaves no byte, so RZE_1 emits
    // only its 2-byte trailer (the original chunk size).
    __syncthreads();
    planes_read(2u);
    if (tid == 0) {
      lookback_publish(sy, sm.epoch, m.c, 2u);
      pend = Pend{m.c, m.item, nw, 2, 0, 1, 1};
      st_small[0] = (uint32_t)osize;
    }
    return false;
  }

  // Segment layout: thread t owns BIT-output words 32t..32t+31.
  // Zero-elimination bitmap (d_ZEencodebyteshort): bit i <-> byte i != 0.
  uint32_t q[32], M[4] = {0, 0, 0, 0};
  auto load8 = [&](int j, uint32_t* x) {
    const uint4* r = reinterpret_cast<const uint4*>(Y + 32 * tid);
    const uint4 a = r[(2 * j) ^ (tid & 7)], b = r[(2 * j + 1) ^ (tid & 7)];
    x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
  };
  if (KEEP) {
    row_load(Y, tid, q);
    uint32_t qany = 0;
#pragma unroll
    for (int k = 0; k < 32; k++) qany |= q[k];
    if (qany) {
#pragma unroll
      for (int j = 0; j < 4; j++) M[j] = nz_bytes8(q + 8 * j);
    }
  } else {
#pragma unroll 1
    for (int j = 0; j < 4; j++) {
      uint32_t x[8];
      load8(j, x);
      M[0] = M[1];
      M[1] = M[2];
      M[2] = M[3];
      M[3] = 0;
      if (x[0] | x[1] | x[2] | x[3] | x[4] | x[5] | x[6] | x[7]) M[3] = nz_bytes8(x);
    }
  }
  const uint32_t nz = __popc(M[0]) + __popc(M[1]) + __popc(M[2]) + __popc(M[3]);
  // Last bitmap byte of the previous segment (RE's predecessor of byte 0).
  uint32_t pb = 0;
  if (tid > 0) {
    const int w = 32 * tid - 2;
    const uint32_t x0 = Y[swz(w)];
    const uint32_t x1 = Y[swz(w + 1)];
    pb = nz_nibble(x0) | (nz_nibble(x1) << 4);
  }
  // Repetition elimination, level 1 (d_REencode4wordsperthread): keep bitmap
  // byte j iff it differs from byte j-1.
  uint32_t K = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t sh = (M[j] << 8) | (j ? (M[j - 1] >> 24) : pb);
    K |= nz_nibble(M[j] ^ sh) << (4 * j);
  }
  const uint32_t c1 = __popc(K);
  sm.l2[tid] = (uint16_t)K;
  uint32_t tot;
  const uint32_t ex = block_scan_excl(nz | (c1 << 16), sm.scan_a, tot);
  const uint32_t NZ = tot & 0xffffu, C1 = tot >> 16;
  const uint32_t zoff = ex & 0xffffu, c1off = ex >> 16;
  planes_read(NZ + C1 + 288 + 6);
  // (barrier inside the scan: the planes have been read)

  // Levels 2 and 3 and the top bitmap (d_REencode1wordperthread) from the
  // 256-byte level-2 bitmap: by warp 0, which publishes the size, and by every
  // warp when only the exact size tells whether the chunk is stored raw.
  bool raw = false;
  const bool close = NZ + C1 + 288 + 6 >= (unsigned)osize;
  const bool small = NZ + C1 + 288 + 6 <= SMALL;
  if (small) st = st_small;
  if (warp == 0 || close) {
    const uint2 b2 = reinterpret_cast<const uint2*>(sm.l2)[lane];
    const uint32_t pprev = __shfl_up_sync(0xffffffffu, b2.y >> 24, 1);
    const uint32_t p0 = lane ? pprev : 0u;
    const uint32_t k2 = nz_nibble(b2.x ^ ((b2.x << 8) | p0)) | (nz_nibble(b2.y ^ ((b2.y << 8) | (b2.x >> 24))) << 4);
    uint32_t C2;
    const uint32_t off2 = warp_scan_excl(__popc(k2), C2);
    const uint32_t p3 = __shfl_up_sync(0xffffffffu, k2, 1);
    const bool keep3 = k2 != (lane ? p3 : 0u);
    const uint32_t top = __ballot_sync(0xffffffffu, keep3);
    const uint32_t C3 = __popc(top);
    const uint32_t off3 = __popc(top & ((1u << lane) - 1u));
    const uint32_t T = NZ + C1 + C2 + C3;
    unsigned int csize = (NZ == 0) ? 2u : T + 6u;
    raw = csize >= (unsigned)osize;
    if (raw) csize = osize;
    if (tid == 0) {
      lookback_publish(sy, sm.epoch, m.c, csize);
      pend = Pend{m.c, m.item, nw, (int)csize, (int)raw, (int)(small && !raw), 1};
    }
    if (warp == 0 && !raw) {
      if (NZ == 0) {
        if (lane < 2) *staged_byte(st, lane, small) = (uint8_t)(osize >> (8 * lane));
      } else {
        // the word that the level-1 bytes end in (no put() completes it)
        if (lane == 0 && !small) st[staged((NZ + C1) >> 2)] = 0;
        __syncwarp();
        uint32_t p = NZ + C1 + off2;
#pragma unroll
        for (int j = 0; j < 8; j++)
          if ((k2 >> j) & 1) *staged_byte(st, p++, small) = (uint8_t)((j < 4 ? b2.x : b2.y) >> (8 * (j & 3)));
        if (keep3) *staged_byte(st, NZ + C1 + C2 + off3, small) = (uint8_t)k2;
        if (lane < 4) *staged_byte(st, T + lane, small) = (uint8_t)(top >> (8 * lane));
        if (lane == 4) *staged_byte(st, T + 4, small) = (uint8_t)osize;
        if (lane == 5) *staged_byte(st, T + 5, small) = (uint8_t)(osize >> 8);
      }
    }
  }
  if (raw) return true;
  // Compaction of the zero-eliminated bytes and the kept level-1 bitmap bytes.
  if (small) {
    // few bytes, not padded: the non-zero words in order, read back from the
    // planes, and the kept bitmap bytes
    uint8_t* sb = reinterpret_cast<uint8_t*>(st);
    uint32_t wm = nz_nibbles8(M[0]) | (nz_nibbles8(M[1]) << 8) | (nz_nibbles8(M[2]) << 16) | (nz_nibbles8(M[3]) << 24);
    uint32_t p = zoff;
    while (wm) {  // bit k: word k has a byte
      const uint32_t k = __ffs(wm) - 1;
      wm &= wm - 1;
      const uint32_t mk = nibble_at(M, k);
      const uint32_t w = Y[swz(32 * tid + k)];
      if (mk & 1u) sb[p] = (uint8_t)w;
      if (mk & 2u) sb[p + (mk & 1u)] = (uint8_t)(w >> 8);
      if (mk & 4u) sb[p + __popc(mk & 3u)] = (uint8_t)(w >> 16);
      if (mk & 8u) sb[p + __popc(mk & 7u)] = (uint8_t)(w >> 24);
      p += __popc(mk);
    }
    if (K) {
      p = NZ + c1off;
#pragma unroll
      for (int j = 0; j < 16; j++)
        if ((K >> j) & 1) sb[p++] = (uint8_t)(M[j >> 2] >> (8 * (j & 3)));
    }
    return false;
  }
  if (__any_sync(0xffffffffu, (nz | K) != 0)) {
    pz = Packer(zoff);
    pk = Packer(NZ + c1off);
    if (KEEP) {
#pragma unroll
      for (int k = 0; k < 32; k++) pz.put(st, q[k], pack_entry(M[k >> 3], k & 7));
#pragma unroll
      for (int j = 0; j < 4; j++) pk.put(st, M[j], pack_entry(K, j));
    } else {
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        uint32_t x[8];
        load8(j, x);
        const uint32_t m4 = M[0];
        M[0] = M[1];
        M[1] = M[2];
        M[2] = M[3];
#pragma unroll
        for (int k = 0; k < 8; k++) pz.put(st, x[k], pack_entry(m4, k));
        pk.put(st, m4, pack_entry(K, 0));
        K >>= 4;
      }
    }
  }
  return false;
}

// A payload from words in global memory (out of line: rare).  INPUT: a raw
// chunk's floats, read again; two blocks in flight, read-only loads: the words
// come from L2 or DRAM (store of 128 MiB of random bits: 110 -> 106 us; four
// blocks: 110).  Else a compressed payload that this CTA has spilled, padded as
// it was staged.
template <bool INPUT>
__device__ __noinline__ void flush_words(uint8_t* dst, const uint32_t* words, int csize) {
  if (INPUT)
    store_payload<2>(dst, csize, [=](int w) -> uint32_t { return 4 * w < csize ? __ldg(words + w) : 0u; });
  else
    store_payload<2>(dst, csize, [=](int w) -> uint32_t { return __ldcg(words + staged(w)); });
}
// A raw chunk that this CTA has spilled (words 16-byte aligned, 16 readable bytes
// behind them): 16-byte loads, shifted by the alignment of dst.
__device__ __noinline__ void flush_raw(uint8_t* dst, const uint32_t* words, int csize) {
  const int tid = threadIdx.x;
  const uint8_t* bytes = reinterpret_cast<const uint8_t*>(words);
  const uint4* w4 = reinterpret_cast<const uint4*>(words);
  const uintptr_t A = reinterpret_cast<uintptr_t>(dst);
  const uintptr_t a0 = (A + 15) & ~uintptr_t(15);
  const uintptr_t a1 = max((A + csize) & ~uintptr_t(15), a0);
  const int head = min((int)(a0 - A), csize), nblk = (int)((a1 - a0) >> 4);
#pragma unroll 2
  for (int b = tid; b < nblk; b += NT) {
    uint4 x = __ldcg(w4 + b), y = __ldcg(w4 + b + 1);
    if (head & 8) x = make_uint4(x.z, x.w, y.x, y.y), y = make_uint4(y.z, y.w, 0u, 0u);
    if (head & 4) x = make_uint4(x.y, x.z, x.w, y.x), y.x = y.y;
    const uint32_t r = 8u * (head & 3);
    *reinterpret_cast<uint4*>(a0 + 16 * (uintptr_t)b) =
        make_uint4(__funnelshift_r(x.x, x.y, r), __funnelshift_r(x.y, x.z, r), __funnelshift_r(x.z, x.w, r),
                   __funnelshift_r(x.w, y.x, r));
  }
  if (tid < head) dst[tid] = __ldcg(bytes + tid);
  const int at = head + 16 * nblk + tid;
  if (at < csize) dst[at] = __ldcg(bytes + at);
}

// Writes out a pending chunk (p; its output offset in sm.payload_off; both
// visible after a barrier) from its staging buffer -- or from raw_words, the
// input's floats, for a raw chunk of the store (FLOATS) -- and
// its size-table entry; the stream's last chunk also sets the stream size.
template <bool FLOATS>
__device__ __forceinline__ void flush_staged(const Ctl& sm, const Pend& p, const uint32_t* st, const uint32_t* st_small,
                                             const uint32_t* raw_words, uint8_t* data_out, uint16_t* table_out,
                                             long long* out_size, long long chunks) {
  const unsigned long long X = sm.payload_off;
  if (FLOATS && p.raw) {
    flush_words<true>(data_out + X, raw_words, p.csize);
  } else {
    if (p.small) st = st_small;
    const uint32_t pad = p.small ? 31 : 5;  // no padding, or staged()
    store_payload(data_out + X, p.csize, [&](int w) -> uint32_t { return st[(uint32_t)w + ((uint32_t)w >> pad)]; });
  }
  if (threadIdx.x == 0) {
    table_out[p.c] = (uint16_t)p.csize;
    if (p.c == chunks - 1) *out_size = HDR + 2 * chunks + (long long)(X + p.csize);
  }
}

}  // namespace cortado
