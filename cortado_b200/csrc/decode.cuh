// The decoders' per-chunk stages (storage decode, init_recv, resi_recv): undo
// RZE_1, BIT_4 and DIFFMS of one 16 KiB chunk in a 128-thread CTA, 32 words
// per thread (the layouts of device.cuh).
//
// What bounds them: the integer pipe (busy 39-44% of the cycles) and the
// barriers between the dependent phases of a chunk, not DRAM (17-38%).  So the
// bitmap levels are rebuilt with byte permutes instead of chains of dependent
// loads, every warp derives the small levels itself, and the payload and the
// planes have a buffer each: two barriers fewer than with one for both, and
// the next payload arrives while this one's planes are turned into floats.
// Instructions per chunk 5,048 -> 3,831 on a field of nearly all zero bins.
// 128 MiB: init_recv 97 -> 65 us (sinusoids with noise, 14% of the size), 121 ->
// 84 (dense, 66%); storage decode 101 -> 69 at 30%; resi_recv 136 -> 85.
// Two threads per 32-word group (16 words each, up to 48 warps per SM instead
// of 24) measured slower (148, 174, 188 us for init_recv): the added warps
// repeat the scans and bitmap levels, and the pipe was the limit already.
#pragma once
#include "kernels.cuh"

namespace cortado {

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(s));
  return r;
}
// Byte-permute selectors of two bitmap nibbles m (the low 4 bits of x) and m'
// (the next 4): each scatters the first popc(m) bytes of a word to the positions
// of m's set bits and zero-fills the others.  Bit i is spread to nibble i, then
// becomes its rank, or 4 + the rank for an unset bit (a byte of the zero
// operand), with one multiply-add; the multiplies run beside the logic pipe.
// prmt reads a selector's low 16 bits only.
__device__ __forceinline__ void spread_sel2(uint32_t x, uint32_t& s0, uint32_t& s1) {
  uint32_t s = (x * 0x1001u) & 0x000f000fu;
  s = (s * 0x41u) & 0x03030303u;
  s = (s * 9u) & 0x11111111u;
  s0 = s * 0x110cu + 0x4444u;
  s1 = (s >> 16) * 0x110cu + 0x4444u;
}
// Largest magnitude of a, |b|, |c| (NaN if any is).
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(fabsf(b)), "f"(fabsf(c)));
  return r;
}

// ---------------------------------------------------------------- RE decode
// Repetition elimination undone for eight bytes: output byte j is the kept
// byte number popc(K & ((2 << j) - 1)) - 1 of the kept bytes that start at
// byte `pos` of P, or the byte before them (zero when first) while no bit of
// K is set yet.  The nine candidate bytes come in with three word loads, and
// byte permutes pick them by the running counts (spread to nibbles and
// prefix-summed with a multiply), instead of eight loads that each depend on
// the one before.
__device__ __forceinline__ void re_expand8(const uint32_t* P, int pos, bool first, uint32_t K, uint32_t& lo,
                                           uint32_t& hi) {
  const int q = pos - 1;
  const uint32_t sh = 8u * (uint32_t)q;  // funnel shifts use the low five bits: 8 * (q & 3)
  const uint32_t* p = P + (q >> 2);
  const uint32_t w0 = p[0], w1 = p[1], w2 = p[2];
  uint32_t a = __funnelshift_r(w0, w1, sh);  // bytes 0..3 (byte 0: the predecessor)
  const uint32_t b = __funnelshift_r(w1, w2, sh);
  const uint32_t c = w2 >> (sh & 31u);  // byte 8
  if (first) a &= 0xffffff00u;
  uint32_t s = (K * 0x1001u) & 0x000f000fu;
  s = (s * 0x41u) & 0x03030303u;
  s = (s * 9u) & 0x11111111u;
  const uint32_t cnt = s * 0x11111111u;  // nibble j: kept bytes among the first j + 1
  lo = prmt(a, b, cnt);
  const uint32_t c4 = (cnt >> 12) & 15u;
  const uint32_t a2 = __funnelshift_rc(a, b, 8 * c4), b2 = __funnelshift_rc(b, c, 8 * c4);
  hi = prmt(a2, b2, (cnt >> 16) - c4 * 0x1111u);
}

// ---------------------------------------------------------------- RZE decode
// Chunks of at most this many zero-eliminated bytes are expanded word by
// non-zero word.
constexpr uint32_t FEW = 512;
constexpr uint32_t QFEW = 4;  // the same for a quarter of a segment
// Where a segment's masks and byte positions (8 words) are handed over: its own
// row of the plane buffer, at a place that spreads over the banks.
__device__ __forceinline__ uint32_t* seg_info(uint32_t* Q, int seg) { return Q + 32 * seg + 8 * (seg & 3); }

enum ChunkKind : int { CHUNK_ZERO = 0, CHUNK_PLANES = 1, CHUNK_RAW = 2 };

// Undoes RZE_1 (d_iRZE, d_RZE.h:127-206) for the chunk whose payload the
// stage's loads brought into P (at byte offset m.d, m.csize bytes): the BIT_4
// output goes to the swizzled plane buffer Q (a partial chunk's in the full
// chunks' places).  Returns CHUNK_PLANES,
// CHUNK_ZERO (all words are zero, also for a chunk that cannot be decoded;
// Q is not written) or CHUNK_RAW (Q holds the words as stored, in the float
// tiles' swizzle).  q_free() runs on every thread before the barrier after
// which Q is written.  Ends with a barrier: P has been read and Q is complete.
//
// Every warp decodes the top bitmap and the two small levels by itself (about
// 90 instructions), so no warp waits for another before the level-1 bitmap
// (warp 0 decoding them for the others took a barrier and left three warps
// idle meanwhile).
// RAW: the chunk may be stored uncompressed (else the caller has seen to such chunks).
template <bool RAW, typename Free>
__device__ __forceinline__ ChunkKind rze_decode(Ctl& sm, const Sync& sy, const StageMeta& m, const uint32_t* P,
                                                uint32_t* Q, Free q_free) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = m.nw;
  const int osize = nw * 4;
  const uint8_t* st = reinterpret_cast<const uint8_t*>(P);
  const int csize = m.csize, d = m.d;
  if (m.bad) {  // corrupt size entry or stream header
    if (tid == 0) latch(sy.status, m.bad == 1 ? DST_CORRUPT : DST_SIZE_MISMATCH);
    q_free();
    __syncthreads();
    return CHUNK_ZERO;
  }
  if (RAW && csize == osize) {  // stored uncompressed: realigned words
    q_free();
    __syncthreads();
#pragma unroll 4
    for (int j = 0; j < 32; j++) {
      const int w = tid + NT * j;
      const int o = d + 4 * w;
      if (w < nw) Q[swz(w)] = __funnelshift_r(P[o >> 2], P[(o >> 2) + 1], 8 * (o & 3));
    }
    __syncthreads();
    return CHUNK_RAW;
  }
  // trailer: top bitmap and the original size
  const int T = csize - 6;
  const uint32_t* tp = P + ((d + T) >> 2);
  const uint32_t tsh = 8u * (uint32_t)(d + T);
  const uint32_t t1 = tp[1];
  const uint32_t top = __funnelshift_r(tp[0], t1, tsh);
  bool ok = (__funnelshift_r(t1, tp[2], tsh) & 0xffffu) == (uint32_t)osize;
  if (csize == 2) {  // trailer only: the BIT_4 output was all zero
    if (!ok && tid == 0) latch(sy.status, DST_CORRUPT);
    q_free();
    __syncthreads();
    return CHUNK_ZERO;
  }
  const int c3 = __popc(top);
  const int b3 = T - c3;
  bool wok = b3 >= 0;
  uint32_t M[4] = {0, 0, 0, 0}, l2lo = 0, l2hi = 0;
  int zbase = 0;
  if (wok) {
    // level 3: lane's byte; level 2: its eight bytes
    const int r3 = __popc(top & (0xffffffffu >> (31 - lane))) - 1;
    const uint32_t l3 = r3 >= 0 ? st[d + b3 + r3] : 0u;
    uint32_t c2;
    const uint32_t e2 = warp_scan_excl(__popc(l3), c2);
    const int b2 = b3 - (int)c2;
    wok = b2 >= 0;
    if (wok) {
      re_expand8(P, d + b2 + (int)e2, e2 == 0, l3, l2lo, l2hi);
      const uint32_t pc = __popc(l2lo) + __popc(l2hi);
      zbase = b2 - (int)__reduce_add_sync(0xffffffffu, pc);
      wok = zbase >= 0;
      if (wok) {
        // this thread's two level-2 bytes and their rank among the level-1 bytes
        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < 8 * warp ? pc : 0u);
        const uint32_t klo = __shfl_sync(0xffffffffu, l2lo, 8 * warp + (lane >> 2));
        const uint32_t khi = __shfl_sync(0xffffffffu, l2hi, 8 * warp + (lane >> 2));
        const uint32_t K = prmt(klo, khi, 0x10u + 0x22u * (lane & 3)) & 0xffffu;
        uint32_t kt;
        const uint32_t rk = before + warp_scan_excl(__popc(K), kt);
        const uint32_t rk2 = rk + __popc(K & 0xffu);
        re_expand8(P, d + zbase + (int)rk, rk == 0, K & 0xffu, M[0], M[1]);
        re_expand8(P, d + zbase + (int)rk2, rk2 == 0, K >> 8, M[2], M[3]);
      }
    }
  }
  ok = ok && wok;
  if (32 * tid + 32 > nw) {  // bitmap bits beyond the chunk must be clear
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int keep = 4 * (nw - 32 * tid) - 32 * j;
      const uint32_t k = keep >= 32 ? 0xffffffffu : keep <= 0 ? 0u : (1u << keep) - 1u;
      if (M[j] & ~k) ok = false;
      M[j] &= k;
    }
  }
  q_free();
  const uint32_t nz = __popc(M[0]) + __popc(M[1]) + __popc(M[2]) + __popc(M[3]);
  uint32_t NZ;
  const uint32_t zoff = block_scan_excl(nz, sm.scan_b, NZ);
  if (!wok || NZ != (uint32_t)zbase) ok = false;
  if (!ok) {
    latch(sy.status, DST_CORRUPT);
    M[0] = M[1] = M[2] = M[3] = 0;
  }
  // ZE decode: scatter the non-zero bytes back into the words.
  if (NZ <= FEW) {
    // few bytes: every thread clears its segment and fills in the non-zero words
    uint32_t* row = Q + 32 * tid;
    const uint32_t xr = tid & 7u;
    uint4* r4 = reinterpret_cast<uint4*>(row);
#pragma unroll
    for (int u = 0; u < 8; u++) r4[u ^ xr] = make_uint4(0, 0, 0, 0);
    uint32_t p = (uint32_t)d + zoff;
#pragma unroll
    for (int part = 0; part < 4; part++) {
      uint32_t m32 = M[part];
      while (m32) {
        const uint32_t b = (__ffs(m32) - 1) & 28u;
        const uint32_t mk = (m32 >> b) & 15u;
        m32 ^= mk << b;
        const uint32_t lo = P[p >> 2], hi = P[(p >> 2) + 1];
        uint32_t s0, s1;
        spread_sel2(mk, s0, s1);
        row[(8 * part + (b >> 2)) ^ (xr << 2)] = prmt(__funnelshift_r(lo, hi, 8 * p), 0u, s0);
        p += __popc(mk);
      }
    }
  } else {
    // The non-zero bytes of real data lie in the low planes, the last segments.
    // So that all warps share them, the segments are expanded 32 at a time, a
    // quarter of one (8 words) per thread; a segment's masks and byte positions
    // pass through its own row of Q.  (With a segment per thread one or two
    // warps did all the work while the others waited at the barrier: 256 MiB,
    // init_recv 137 -> 133 us at 6% of the size, resi_send 310 -> 303 us.  The
    // same split of the encoders' packing cost as much as it gave.)
    {
      uint4* info = reinterpret_cast<uint4*>(seg_info(Q, tid));
      info[0] = make_uint4(M[0], M[1], M[2], M[3]);
      const uint32_t p0 = (uint32_t)d + zoff, p1 = p0 + __popc(M[0]), p2 = p1 + __popc(M[1]);
      info[1] = make_uint4(p0, p1, p2, p2 + __popc(M[2]));
    }
    __syncthreads();
    const uint32_t quarter = tid & 3, rot = (tid >> 2) & 3;  // quarters start at different words (banks)
#pragma unroll 1
    for (int seg = tid >> 2; seg < NT; seg += 32) {
      const uint32_t* info = seg_info(Q, seg) + quarter;
      uint32_t m = info[0], p = info[4];
      uint32_t* row = Q + 32 * seg;
      const uint32_t x = ((seg & 7) << 2) ^ (8 * quarter);  // word k of the quarter: row[k ^ x]
      const uint32_t n = __popc(m);
      if (__any_sync(0xffffffffu, n > QFEW)) {  // (also: the warp has read its segments' masks)
        const uint32_t R = __funnelshift_r(m, m, 8 * rot);
        p += rot ? __popc(m & ((1u << (8 * rot)) - 1u)) : n;
        uint32_t k = 2 * rot;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (k == 0) p -= n;  // back to the quarter's first bytes
          const uint32_t mk = prmt(R, 0u, 0x4440u | j);
          uint32_t s0, s1;
          spread_sel2(mk, s0, s1);
          const uint32_t* w = reinterpret_cast<const uint32_t*>(st + (p & ~3u));
          uint2 q;
          q.x = prmt(__funnelshift_r(w[0], w[1], 8 * p), 0u, s0);
          p += __popc(mk & 15u);
          w = reinterpret_cast<const uint32_t*>(st + (p & ~3u));
          q.y = prmt(__funnelshift_r(w[0], w[1], 8 * p), 0u, s1);
          p += __popc(mk >> 4);
          *reinterpret_cast<uint2*>(row + (k ^ x)) = q;
          k = (k + 2) & 6u;
        }
      } else {  // few bytes: clear the quarter, fill in the non-zero words
        uint4* r4 = reinterpret_cast<uint4*>(row);
        r4[(2 * quarter) ^ (seg & 7)] = make_uint4(0, 0, 0, 0);
        r4[(2 * quarter + 1) ^ (seg & 7)] = make_uint4(0, 0, 0, 0);
        while (m) {
          const uint32_t b = (__ffs(m) - 1) & 28u;
          const uint32_t mk = (m >> b) & 15u;
          m ^= mk << b;
          const uint32_t* w = reinterpret_cast<const uint32_t*>(st + (p & ~3u));
          uint32_t s0, s1;
          spread_sel2(mk, s0, s1);
          row[(b >> 2) ^ x] = prmt(__funnelshift_r(w[0], w[1], 8 * p), 0u, s0);
          p += __popc(mk);
        }
      }
    }
  }
  __syncthreads();
  if (nw != CW) widen_planes(Q, nw);
  return CHUNK_PLANES;
}

}  // namespace cortado
