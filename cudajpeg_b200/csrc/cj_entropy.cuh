// cj_entropy.cuh -- device building blocks of the entropy decode in the
// persistent batch kernel (batch.cu): destuff classification, subsequence
// lanes, speculative block decode, the warp settle loop and the cooperative
// coefficient write-out.
#pragma once
#include <limits.h>
#include <stddef.h>
#include <stdint.h>

#include "cj_core.h"
#include "cj_scan_util.cuh"

// 16 stuffed bytes starting at `base`, their neighbours, and what to keep.
struct CJChunk {
  uint32_t w[4];    // the 16 bytes, little-endian words
  uint32_t keep;    // bit j: byte j is entropy data
  uint32_t mark;    // bit j: byte j is the FF of an RSTn marker
  uint32_t next;    // byte after the chunk (marker code of bit 15)
  bool bad;         // an FF followed by anything but 00 / D0-D7
};

__device__ __forceinline__ uint32_t cj_byte(const CJChunk& c, int j) {
  return (c.w[j >> 2] >> (8 * (j & 3))) & 0xFF;
}

// The memory a chunk is classified from: the two aligned 16-byte words
// around its 16 bytes and the one after them, and the byte before it.  For a
// chunk that starts inside the data (base < n) the words lie below
// raw + n + 31; the callers' buffers hold at least 31 bytes past the data and
// start on a 16-byte boundary.  Loaded apart from the classification so that
// a loop can fetch its next chunk early.
struct CJChunkIn {
  uint4 lo, hi;
  uint32_t sh;    // the chunk's offset inside lo
  uint32_t prev;  // the byte before the chunk (0 at the start)
};

__device__ __forceinline__ CJChunkIn cj_chunk_load(const uint8_t* raw, int64_t n, int64_t base) {
  CJChunkIn x;
  x.lo = x.hi = make_uint4(0, 0, 0, 0);
  x.sh = 0;
  if (base < n) {
    const uintptr_t addr = (uintptr_t)(raw + base);
    const uint4* q = reinterpret_cast<const uint4*>(addr & ~(uintptr_t)15);
    x.lo = q[0];
    x.hi = q[1];
    x.sh = (uint32_t)(addr & 15);
  }
  x.prev = (base > 0 && base - 1 < n) ? raw[base - 1] : 0;
  return x;
}

// Classify a loaded chunk: its bytes come out of the two words by funnel
// shifts, whatever its alignment; bytes at or past n read as 0.
__device__ __forceinline__ CJChunk cj_classify_in(const CJChunkIn& x, int64_t n, int64_t base) {
  CJChunk c;
  c.keep = c.mark = 0;
  c.bad = false;
  c.w[0] = c.w[1] = c.w[2] = c.w[3] = 0;
  c.next = 0;
  if (base < n) {
    const uint4 lo = x.lo, hi = x.hi;
    const uint32_t sh = x.sh, bs = (sh & 3) * 8;
    uint32_t a0, a1, a2, a3, a4, a5;
    switch (sh >> 2) {
      case 0: a0 = lo.x; a1 = lo.y; a2 = lo.z; a3 = lo.w; a4 = hi.x; a5 = hi.y; break;
      case 1: a0 = lo.y; a1 = lo.z; a2 = lo.w; a3 = hi.x; a4 = hi.y; a5 = hi.z; break;
      case 2: a0 = lo.z; a1 = lo.w; a2 = hi.x; a3 = hi.y; a4 = hi.z; a5 = hi.w; break;
      default: a0 = lo.w; a1 = hi.x; a2 = hi.y; a3 = hi.z; a4 = hi.w; a5 = 0; break;
    }
    c.w[0] = __funnelshift_r(a0, a1, bs);
    c.w[1] = __funnelshift_r(a1, a2, bs);
    c.w[2] = __funnelshift_r(a2, a3, bs);
    c.w[3] = __funnelshift_r(a3, a4, bs);
    // byte 16 of the chunk: byte 0 of the next word
    const uint32_t after = __funnelshift_r(a4, a5, bs) & 0xFF;
    c.next = (base + 16 < n) ? after : 0;
    if (base + 16 > n) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int64_t valid = n - (base + 4 * k);  // bytes of word k below n
        if (valid <= 0) c.w[k] = 0;
        else if (valid < 4) c.w[k] &= (1u << (8 * valid)) - 1u;
      }
    }
  }
  uint32_t prev = x.prev;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    if (base + j >= n) break;
    uint32_t b = cj_byte(c, j);
    uint32_t nx = (j < 15) ? cj_byte(c, j + 1) : c.next;
    bool has_next = base + j + 1 < n;
    if (prev == 0xFF && (base + j) > 0) {
      // second byte of an FF pair: stuffing or the RSTn code, never data
      if (b != 0x00 && (b & 0xF8) != 0xD0) c.bad = true;
    } else if (b == 0xFF) {
      if (has_next && nx == 0x00) c.keep |= 1u << j;
      else if (has_next && (nx & 0xF8) == 0xD0) c.mark |= 1u << j;
      else c.bad = true;
    } else {
      c.keep |= 1u << j;
    }
    prev = b;
  }
  return c;
}

struct CJLane {
  uint64_t begin, end;   // this subsequence's bits
  uint64_t end_byte;     // its segment's end (bytes)
  int seg;
  bool head, last, active;
};

__device__ __forceinline__ CJLane cj_lane(const CJSegment* segs, int nseg, int nsub, int i,
                                          int sub_bits) {
  CJLane l;
  l.active = i < nsub;
  l.begin = l.end = l.end_byte = 0;
  l.seg = 0;
  l.head = l.last = false;
  if (!l.active) return l;
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (segs[mid].first_sub <= i) lo = mid;
    else hi = mid - 1;
  }
  const CJSegment& s = segs[lo];
  int j = i - s.first_sub;
  l.seg = lo;
  l.begin = s.bit_begin + (uint64_t)j * sub_bits;
  l.end = min(s.bit_end, l.begin + (uint64_t)sub_bits);
  if (l.begin > s.bit_end) l.begin = s.bit_end;
  l.end_byte = s.bit_end >> 3;
  l.head = (j == 0);
  l.last = (j == s.nsub - 1);
  return l;
}

// Shared memory by its 32-bit address: the decode loops are not inlined, and a
// pointer passed to them would be accessed as a generic one.  cj_tab16 reads a
// table that does not change while the loop runs, so it may be scheduled
// freely.
__device__ __forceinline__ uint32_t cj_lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t cj_tab16(uint32_t a) {
  uint16_t v;
  asm("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
// An entry of a CJSpecTab: in shared memory at address a, or (GLOBAL) a bytes into
// the set at `set` in global memory.
template <bool GLOBAL>
__device__ __forceinline__ uint32_t cj_entry(const uint8_t* set, uint32_t a) {
  if (!GLOBAL) return cj_tab16(a);
  uint16_t v;
  asm("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(set + a));
  return v;
}
__device__ __forceinline__ uint32_t cj_tab8(uint32_t a) {
  uint32_t v;
  asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ CJDone cj_lds_done(uint32_t a) {
  CJDone v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.block), "=r"(v.lane) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cj_sts_done(uint32_t a, CJDone v) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(v.block), "r"(v.lane) : "memory");
}
__device__ __forceinline__ uint4 cj_lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cj_sts128_zero(uint32_t a) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(a), "r"(0u) : "memory");
}
__device__ __forceinline__ void cj_sts16(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void cj_sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Bit window of a lane in the warp-synchronous decode loops.  A lane's
// stream runs through a ring of WORDS big-endian words in shared
// memory (word w in slot w mod WORDS, `col` + 128 bytes per slot: one
// bank per lane, so every access is conflict-free at any progress of the
// lanes).  The current and the next word are in registers and the one after
// them is read a symbol ahead, without branches: a symbol's chain is a funnel
// shift, the table lookup, the position update and two selects.  Global memory
// is touched only in refill(), which the whole warp runs together every
// ROUNDS rounds of the loop: a 16-byte chunk fetched there has until
// the next refill to arrive.
// Bytes at or past `end_byte` read as 0xFF (the padding the reference's bit
// reader supplies); memory past them is not relied on.
#define CJ_STEPS_PER_ROUND 3
// A round is three symbols of at most 31 bits: at most 3 words.  With 2 words
// read ahead and up to 3 of the oldest chunk passed, 16 words serve 3 rounds,
// and 8 words one (the word read ahead after a round of 3 crossings is read
// again by the refill).
#define CJ_RING_WORDS 16
#define CJ_RING_ROUNDS 3
#define CJ_WRITE_WORDS 8
template <int WORDS>
struct CJWin {
  const uint4* chunks;    // the image's destuffed data, 16-byte aligned
  uint32_t col;           // this lane's ring column (shared address)
  uint32_t end_byte, cb;  // chunks cb .. cb + 3 are in the ring, cb + 4 in pf
  uint4 pf;
  uint32_t cur, nxt, nn, pos;  // words pos / 32, + 1, + 2; the next bit

  __device__ __forceinline__ uint4 load(uint32_t c) const {
    return 16u * c < end_byte ? chunks[c] : make_uint4(0, 0, 0, 0);
  }
  __device__ __forceinline__ void put(uint32_t c, uint4 v) {
    uint32_t w[4] = {cj_bswap(v.x), cj_bswap(v.y), cj_bswap(v.z), cj_bswap(v.w)};
    const uint32_t first = 16u * c;
    if (first + 16 > end_byte) {  // the last chunks of a segment
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int valid = (int)(end_byte - first) - 4 * i;  // data bytes of word i
        if (valid <= 0) w[i] = 0xFFFFFFFFu;
        else if (valid < 4) w[i] |= 0xFFFFFFFFu >> (8 * valid);
      }
    }
    const uint32_t o = col + 128 * ((4 * c) & (WORDS - 1));
#pragma unroll
    for (int i = 0; i < 4; i++) cj_sts32(o + 128 * i, w[i]);
  }
  // word pos / 32 + ahead
  __device__ __forceinline__ uint32_t word(uint32_t ahead) const {
    return cj_lds32(col + (((pos + 32 * ahead) << 2) & (128 * (WORDS - 1))));
  }
  __device__ __forceinline__ void init(const uint4* data, uint32_t ring_col, uint32_t eb, uint32_t p) {
    chunks = data;
    col = ring_col;
    end_byte = eb;
    cb = p >> 7;
    uint4 v[WORDS / 4];
#pragma unroll
    for (int i = 0; i < WORDS / 4; i++) v[i] = load(cb + i);
    pf = load(cb + WORDS / 4);
#pragma unroll
    for (int i = 0; i < WORDS / 4; i++) put(cb + i, v[i]);
    pos = p;
    cur = word(0);
    nxt = word(1);
    nn = word(2);
  }
  // Replace the chunks the window has left behind.
  __device__ __forceinline__ void refill() {
    while ((pos >> 7) > cb) {
      put(cb + WORDS / 4, pf);
      cb++;
      pf = load(cb + WORDS / 4);
      if (WORDS == 8) nn = word(2);  // read before its chunk was there, after 3 crossings
    }
    if (WORDS == 8) cj_fold_position(pos, cb);  // (the write-out's)
  }
  __device__ __forceinline__ uint32_t peek() const { return __funnelshift_l(nxt, cur, pos); }
  // u <= 31: at most one word is crossed
  __device__ __forceinline__ void skip(uint32_t u) {
    const uint32_t np = pos + u;
    const bool cross = ((pos ^ np) & 32) != 0;
    cur = cross ? nxt : cur;
    nxt = cross ? nn : nxt;
    pos = np;
    nn = word(2);
  }
};

// Checkpoints of a subsequence decode: the decoder state at the first block
// boundary at or after each of CJ_CKPTS thresholds (1/4, 1/2, 3/4 of the
// subsequence): position relative to the subsequence start and MCU phase
// (pp = phase << 24 | position), blocks begun before it, DC sums before it.
// Thresholds the decode never passes get its exit state.
#define CJ_CKPTS 3
struct CJCkpt {
  uint32_t pp;
  int32_t nb, d0, d1, d2;
};

// The decode under way joined an earlier decode of the same subsequence: the
// two coincide from the block boundary at checkpoint `j` on.
struct CJJoin {
  int j;    // CJ_CKPTS: no join
  int src;  // -1: the lane's own previous decode, else hypothesis src
};

// Speculative decode of one subsequence per lane, from `start`, by a whole
// warp (lanes with run = false take part in the votes only): blocks beginning
// before the subsequence's end, their DC sums, and the state after them.
//
// The loop is straight-line code over the tables of CJSpecTab: a divergent
// branch costs some 40 cycles whether one lane takes it or all, and with 32
// lanes at different symbols every branch is taken by some lane in almost
// every step (measured on 4:2:0 photos: 870 cycles per symbol step with branches
// for word crossings, long codes and block ends, 280 as here; the sync phase of
// the 1024-image mix 0.88 -> 0.42 ms, of 48 1080p frames 1.05 -> 0.33 ms).  So word crossings are selects, a long code
// is two steps (its prefix entry makes its subtable the next step's table), a
// lane whose block has ended consumes nothing, and the end of blocks is one
// branch per round of three steps.  The DC entry and window are kept and the
// difference added when the block ends.  On a valid stream this is the serial
// T.81 block decode (src/decodeScanGPU.cu:78-100) symbol for symbol; after a
// symbol that fails, the block is counted and decoding goes on behind it (the
// write-out reports the block).
//
// Checkpoints (`ck`, CJ_CKPTS of them) are written for every decode.  A
// re-decode (`resume`) from a corrected start compares each checkpoint it
// reaches with those of the previous decode `x.r`: when position and phase agree
// the two decodes are identical from there on, so it stops and takes the
// previous totals shifted by the difference in blocks and DC sums before that
// point (shifting the later checkpoints too).  The result equals a full
// decode from `start`.  HYP: the same test against the `nh` hypothesis decodes
// of the subsequence, whose checkpoint positions lie in shared memory (`hpp`,
// column of cj_hyp_fill).  The tests read registers and shared memory only and
// the totals of all joined lanes are taken together after the loop: lanes
// reach their checkpoints at different steps, so a global load there would
// stall the warp once per lane and checkpoint.
// Phase entries: per MCU phase the shared addresses of the phase's tables
// (x: dc | acm << 16), then ac1, the component << 16 and the next phase << 24
// (y).  Written by the whole warp for an image and its tables at `tab` (0: offsets
// into the set, for tables in global memory).
__device__ __forceinline__ void cj_phase_entries(const CJScanParams& sp, uint32_t tab, uint32_t phases) {
  const int i = threadIdx.x & 31, bpm = sp.bpm;
  __syncwarp();
  if (i < bpm) {
    const uint32_t c = sp.phase_comp[i], d = sp.comp_dc[c], a = sp.comp_ac[c] - 2u;
    const uint32_t dc = tab + (uint32_t)offsetof(CJSpecTab, dc) + d * (uint32_t)sizeof(CJSpecTab::dc[0]);
    const uint32_t ac1 = tab + (uint32_t)offsetof(CJSpecTab, ac1) + a * (uint32_t)sizeof(CJSpecTab::ac1[0]);
    const uint32_t acm = tab + a * (uint32_t)sizeof(CJSpecTab::acm[0]);
    cj_sts32(phases + 8 * i, dc | (acm << 16));
    cj_sts32(phases + 8 * i + 4, ac1 | (c << 16) | ((i + 1 == bpm ? 0u : (uint32_t)i + 1) << 24));
  }
  __syncwarp();
}
// from an ac1 table to the subtables of its long codes
static_assert(sizeof(CJSpecTab::sub[0]) == sizeof(CJSpecTab::ac1[0]), "sub follows ac1 at one distance");
#define CJ_SPEC_SUB ((uint32_t)(offsetof(CJSpecTab, sub) - offsetof(CJSpecTab, ac1)))

// A warp's shared memory in the speculative decode.
struct CJSpecWarp {
  uint32_t ring[CJ_RING_WORDS][32];
  uint2 phase[CJ_MAX_BPM];
};

// One lane's part of a decode: where and how (all lanes of the warp agree on
// sp, tp, tab), and its record in and out.
struct CJSpecJob {
  const CJScanParams *sp, *tp;
  const uint4* data;
  const uint8_t* gtab;             // the CJSpecTab where it is not in shared memory (tab: 0)
  uint32_t tab, ring, phase, hpp;  // shared addresses: CJSpecTab, ring column, phase entries, hypothesis column
  uint32_t begin, end, end_byte, cstep;
  int nh;
  bool resume;  // r and ck hold an earlier decode of the subsequence
  CJCkpt* ck;
  const CJCkpt* hck;
  const CJSubRec* hrec;
  CJSubRec r;
};
__device__ __forceinline__ void cj_spec_job(CJSpecJob& x, const CJScanParams& sp, const CJScanParams& tp,
                                            uint32_t tab, const uint8_t* gtab, const void* data, const CJLane& ln,
                                            CJCkpt* ck, uint32_t cstep, const CJSpecWarp& sw) {
  x.sp = &sp;
  x.tp = &tp;
  x.tab = tab;
  x.gtab = gtab;
  x.data = reinterpret_cast<const uint4*>(data);
  x.begin = (uint32_t)ln.begin;
  x.end = (uint32_t)ln.end;
  x.end_byte = (uint32_t)ln.end_byte;
  x.ck = ck;
  x.cstep = cstep;
  x.ring = (uint32_t)__cvta_generic_to_shared(sw.ring) + 4 * (threadIdx.x & 31);
  x.phase = (uint32_t)__cvta_generic_to_shared(sw.phase);
  x.nh = 0;
  x.resume = false;
}

// Not inlined: in a function of its own the loop has the kernel's whole
// register budget, and the phases around it keep their state across the call
// in local memory instead of squeezing the loop (550 bytes of spills, some in
// the loop, when inlined at 64 registers).
template <bool HYP, bool GLOBAL>
__device__ __noinline__ void cj_spec_warp(CJSpecJob* job, bool run, uint64_t start) {
  CJSpecJob& x = *job;
  const uint8_t* const set = x.gtab;
  CJWin<CJ_RING_WORDS> br;
  const uint32_t begin = x.begin, end = x.end, cstep = x.cstep, phases = x.phase;
  CJCkpt* const ck = x.ck;
  const int bpm = x.sp->bpm;
  cj_phase_entries(*x.sp, x.tab, phases);
  int c = 0, k = -1, nb = 0, d0 = 0, d1 = 0, d2 = 0, j = 0;
  uint32_t dcv = 0, dce = 0, thresh = cstep;
  uint32_t next = cj_state_phase(start);  // phase of the block after the current one
  uint32_t tab = x.tab, sh = 32 - CJ_MULTI_DC_BITS, acm = x.tab, ac1 = x.tab;
  uint2 ph = make_uint2(cj_lds32(phases + 8 * next), cj_lds32(phases + 8 * next + 4));  // entry of phase `next`
  br.pos = (uint32_t)cj_state_bit(start);
  br.col = x.ring;
  br.cur = br.nxt = br.nn = 0;
  uint32_t old[CJ_CKPTS];
  CJJoin jn = {CJ_CKPTS, -1};
#pragma unroll
  for (int q = 0; q < CJ_CKPTS; q++) old[q] = 0xFFFFFFFFu;  // matches no decode state
  // checkpoints may have been written by another SM in an earlier pass of
  // the same kernel: read them from L2, never a stale L1 line
  if (run && x.resume) {
#pragma unroll
    for (int q = 0; q < CJ_CKPTS; q++) old[q] = __ldcg(&ck[q].pp);
  }
  auto phase = [&]() { return next ? next - 1 : (uint32_t)bpm - 1; };  // of the current block
  // Begin the block of phase `next`.
  auto begin_block = [&]() {
    tab = ph.x & 0xFFFFu;
    sh = 32 - CJ_MULTI_DC_BITS;
    acm = ph.x >> 16;
    ac1 = ph.y & 0xFFFFu;
    c = (int)((ph.y >> 16) & 255);
    next = ph.y >> 24;
    ph.x = cj_lds32(phases + 8 * next);
    ph.y = cj_lds32(phases + 8 * next + 4);
    k = -1;
  };
  // The checkpoints at the block boundary `rel` bits into the subsequence;
  // true when this decode has joined an earlier one.
  auto checkpoint = [&](uint32_t rel) -> bool {
    const uint32_t pp = (phase() << 24) | rel;
    while (j < CJ_CKPTS && rel >= thresh) {
      uint32_t o = old[0];
#pragma unroll
      for (int q = 1; q < CJ_CKPTS; q++) o = j == q ? old[q] : o;
      int src = o == pp ? -1 : -2;
      if (HYP)
        for (int h = 0; src == -2 && h < x.nh; h++)
          if (cj_lds32(x.hpp + 128 * (h * CJ_CKPTS + j)) == pp) src = h;
      if (src != -2) {
        jn.j = j;
        jn.src = src;
        return true;
      }
      ck[j] = CJCkpt{pp, nb, d0, d1, d2};
      j++;
      thresh += cstep;
    }
    return false;
  };
  bool live = run && br.pos < end;
  if (live) br.init(x.data, x.ring, x.end_byte, br.pos);
  begin_block();
  if (live && br.pos - begin >= thresh) live = !checkpoint(br.pos - begin);
  // Consume entry st and choose the next step's table.
  auto apply = [&](uint32_t st) {
    br.skip(st & 31);
    k += (int)(st >> 9);
    const bool prefix = st < (1u << 9);
    const bool high = k > CJ_MULTI_MAXK;
    tab = prefix ? ac1 + CJ_SPEC_SUB + ((st & 0x1E0u) << 2) : (high ? ac1 : acm);
    sh = prefix ? 26 : (high ? 32 - CJ_FAST_BITS : 32 - CJ_MULTI_BITS);
  };
  uint32_t p = br.pos;  // the last block boundary
  while (__any_sync(CJ_FULL, live)) {
    if (live) br.refill();
    __syncwarp();
#pragma unroll 1
    for (int u = 0; u < CJ_RING_ROUNDS; u++) {
#pragma unroll
      for (int q = 0; q < CJ_STEPS_PER_ROUND; q++) {
        const uint32_t v = br.peek();
        uint32_t st = cj_entry<GLOBAL>(set, tab + 2 * (v >> sh));
        if (q == 0) {  // a DC symbol can only come first in a round
          dcv = k < 0 ? v : dcv;
          dce = k < 0 ? st : dce;
        }
        // (finished lanes decode on behind their end in the first step: their
        // results are taken already)
        if (q > 0) st = k < 63 ? st : 0;
        apply(st);
      }
      if (live && k >= 63) {
        if (k >= CJ_SPEC_FARK) {  // rare
          k -= (int)(CJ_SPEC_FAR >> 9);
          const uint32_t v = br.peek();
          const uint32_t slot = k < 0 ? x.sp->comp_dc[c] : x.sp->comp_ac[c];
          const uint32_t st = cj_spec_entry(cj_step_canonical(x.tp->huff[slot], slot, v), 0, k < 0);
          if (k < 0) {
            dcv = v;
            dce = st;
          }
          apply(st);
        }
        if (k >= 63) {
          const uint32_t size = (dce >> 5) & 15, w = dcv << ((dce & 31) - size);
          // (T.81 F.2.2.1: a magnitude whose first bit is 0 is negative)
          int dd = (int)__funnelshift_rc(w, 0u, 32 - size);
          dd -= (int)w >= 0 ? (int)((1u << size) - 1u) : 0;
          if (c == 0) d0 += dd;
          else if (c == 1) d1 += dd;
          else d2 += dd;
          nb++;
          begin_block();
          p = br.pos;
          if (p >= end) live = false;
          else if (p - begin >= thresh && j < CJ_CKPTS) live = !checkpoint(p - begin);
        }
      }
      __syncwarp();
    }
  }
  const uint32_t m = phase();
  if (!run) return;
  CJSubRec& r = x.r;
  r.start = start;
  if (jn.j == CJ_CKPTS) {
    // thresholds not reached: the exit
    const uint32_t pp = (m << 24) | (p - begin);
#pragma unroll
    for (int q = 0; q < CJ_CKPTS; q++)
      if (q >= j) ck[q] = CJCkpt{pp, nb, d0, d1, d2};
    r.exit = cj_state(p, m);
    r.nblocks = nb;
    r.dc[0] = d0;
    r.dc[1] = d1;
    r.dc[2] = d2;
    return;
  }
  const CJCkpt* sc = HYP && jn.src >= 0 ? x.hck + jn.src * CJ_CKPTS : ck;
  const CJCkpt at = {0, __ldcg(&sc[jn.j].nb), __ldcg(&sc[jn.j].d0), __ldcg(&sc[jn.j].d1), __ldcg(&sc[jn.j].d2)};
  if (HYP && jn.src >= 0) {
    const CJSubRec* hr = x.hrec + jn.src;
    r.exit = __ldcg(&hr->exit);
    r.nblocks = __ldcg(&hr->nblocks);
#pragma unroll
    for (int q = 0; q < 3; q++) r.dc[q] = __ldcg(&hr->dc[q]);
  }
  r.nblocks += nb - at.nb;
  r.dc[0] += d0 - at.d0;
  r.dc[1] += d1 - at.d1;
  r.dc[2] += d2 - at.d2;
#pragma unroll
  for (int q = 0; q < CJ_CKPTS; q++) {
    if (q < jn.j) continue;
    ck[q] = CJCkpt{__ldcg(&sc[q].pp), __ldcg(&sc[q].nb) + nb - at.nb, __ldcg(&sc[q].d0) + d0 - at.d0,
                   __ldcg(&sc[q].d1) + d1 - at.d1, __ldcg(&sc[q].d2) + d2 - at.d2};
  }
}

// GLOBAL: the job's tables may be in global memory (warp-uniform).
template <bool HYP, bool GLOBAL>
__device__ __forceinline__ void cj_spec_run(CJSpecJob& x, bool run, uint64_t start) {
  if (GLOBAL && x.gtab) cj_spec_warp<HYP, GLOBAL>(&x, run, start);
  else cj_spec_warp<HYP, false>(&x, run, start);
}

// The checkpoint positions of a lane's `nh` hypothesis decodes into its
// column of shared memory (entry 32 * (h * CJ_CKPTS + j)).
__device__ __forceinline__ void cj_hyp_fill(uint32_t* hpp, const CJCkpt* hck, int nh) {
#pragma unroll 4
  for (int q = 0; q < nh * CJ_CKPTS; q++) hpp[32 * q] = __ldcg(&hck[q].pp);
}

// Checkpoints of global lane `i` and the threshold spacing of a subsequence.
__device__ __forceinline__ CJCkpt* cj_lane_ckpts(CJCkpt* base, int64_t i) { return base + i * CJ_CKPTS; }
__device__ __forceinline__ uint32_t cj_ckpt_step(int sub_bits) { return (uint32_t)sub_bits / (CJ_CKPTS + 1); }

// Re-decode lanes whose input state (lane 0: `lane0_in`; others: the exit of
// the previous lane) differs from the state they last decoded from, until no
// lane changes.  Lane l settles after at most l+1 re-decodes.
template <bool GLOBAL>
__device__ __forceinline__ bool cj_warp_settle(CJSpecJob& x, const CJLane& ln, uint64_t lane0_in) {
  int lane = threadIdx.x & 31;
  bool dirty = false;
  x.resume = true;
  for (int it = 0; it < 34; it++) {
    uint64_t pred = __shfl_up_sync(CJ_FULL, x.r.exit, 1);
    uint64_t want = ln.head ? x.r.start : (lane == 0 ? lane0_in : pred);
    bool change = ln.active && want != x.r.start;
    if (!__any_sync(CJ_FULL, change)) break;
    cj_spec_run<false, GLOBAL>(x, change, want);
    dirty = dirty || change;
  }
  return dirty;
}

// Errors are ordered by the block they occur in; the status keeps the first
// (stored complemented so an all-zero status means "no error").
__device__ __forceinline__ void cj_raise(CJStatus* st, int64_t block, int code) {
  unsigned long long key = ((unsigned long long)block << 8) | (unsigned)code;
  atomicMax(&st->err_key, ~key);
}

__device__ __forceinline__ void cj_raise_dec(CJStatus* st, int64_t block, int code) {
  unsigned long long key = ((unsigned long long)block << 8) | (unsigned)code;
  atomicMax(&st->dec_err_key, ~key);
}

// Segmented-sum operator over (head flag, sums).
struct CJAgg5 {
  int f, n, a, b, c;
};
__device__ __forceinline__ CJAgg5 cj_op(const CJAgg5& x, const CJAgg5& y) {
  CJAgg5 r;
  r.f = x.f | y.f;
  if (y.f) {
    r.n = y.n; r.a = y.a; r.b = y.b; r.c = y.c;
  } else {
    r.n = x.n + y.n; r.a = x.a + y.a; r.b = x.b + y.b; r.c = x.c + y.c;
  }
  return r;
}

// Segmented exclusive prefix, over the lanes of a warp, of each lane's blocks
// and DC sums: from the last segment head at or before the lane, plus the
// carry from earlier warps (cn, c0..c2) when the segment began before this warp.
__device__ __forceinline__ void cj_warp_prefix(const CJSubRec& r, const CJLane& ln, int cn, int c0,
                                               int c1, int c2, int64_t* blocks, int* d0, int* d1,
                                               int* d2) {
  const int lane = threadIdx.x & 31;
  // Segmented exclusive prefix of (blocks, DC sums) over the warp.
  int s0 = r.nblocks, s1 = r.dc[0], s2 = r.dc[1], s3 = r.dc[2];
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int t0 = __shfl_up_sync(CJ_FULL, s0, d), t1 = __shfl_up_sync(CJ_FULL, s1, d);
    int t2 = __shfl_up_sync(CJ_FULL, s2, d), t3 = __shfl_up_sync(CJ_FULL, s3, d);
    if (lane >= d) {
      s0 += t0; s1 += t1; s2 += t2; s3 += t3;
    }
  }
  unsigned heads = __ballot_sync(CJ_FULL, ln.active && ln.head);
  unsigned mine = heads & ((2u << lane) - 1u);  // heads at or before this lane
  int a = mine ? 31 - __clz(mine) : 0;
  int src = a > 0 ? a - 1 : 0;
  int b0 = __shfl_sync(CJ_FULL, s0, src), b1 = __shfl_sync(CJ_FULL, s1, src);
  int b2 = __shfl_sync(CJ_FULL, s2, src), b3 = __shfl_sync(CJ_FULL, s3, src);
  if (a == 0) b0 = b1 = b2 = b3 = 0;
  int e0 = s0 - r.nblocks - b0, e1 = s1 - r.dc[0] - b1, e2 = s2 - r.dc[1] - b2,
      e3 = s3 - r.dc[2] - b3;
  if (!mine) {
    e0 += cn; e1 += c0; e2 += c1; e3 += c2;
  }
  *blocks = e0;
  *d0 = e1;
  *d1 = e2;
  *d2 = e3;
}

// Blocks lane `ln` writes from block `first`: to its block count, or to its
// segment's last block for the segment's last lane; clamped to the segment.
__device__ __forceinline__ int64_t cj_lane_write_end(const CJLane& ln, const CJSegment& seg, const CJSubRec& r,
                                                     int64_t first) {
  const int64_t bend = seg.first_block + seg.nblocks;
  const int64_t end = ln.last ? bend : first + r.nblocks;
  return end > bend ? bend : end;
}

// A warp's shared memory in the write-out.
struct CJWriteWarp {
  uint32_t ring[CJ_WRITE_WORDS][32];
  uint2 phase[CJ_MAX_BPM];
  CJDone order[32];  // completed blocks of a round
};

// One lane's unit of the write-out (sp .. coef agree over the warp).
struct CJWriteJob {
  const CJScanParams *sp, *tp;
  CJStatus* st;
  const uint4* data;
  int16_t* coef;  // of block `base`
  int64_t base;   // blk and bend count from here
  const uint8_t* gtab;  // as in CJSpecJob
  uint32_t tab, ring, phase, order, wbuf, zz;  // shared addresses (wbuf: the warp's 32 blocks; zz: 2 x zig-zag index)
  uint32_t end_byte, end, stop, seg_end;       // bits: of the subsequence, of the unit, of the segment
  uint32_t pos, m;                             // the unit's first block
  int blk, bend, dc[3];
  bool last, marker;  // the segment's last subsequence; an RSTn follows the segment
  bool cut;           // out: stopped inside block blk at an error
};

// Warp-cooperative write-out of 32 units (one per lane; `active` = false for
// lanes without one), symbol for symbol the serial block decode with the
// same structural checks, as straight-line rounds of three symbols (see
// cj_spec_warp).  Each lane builds its current block in its own 64-entry int16
// buffer in shared memory (all zero on entry and on return; the 16-byte chunks
// of lane l are permuted by l mod 8, so equal positions of different lanes fall
// into different banks).  After every round the warp stores the blocks its
// lanes completed: 8 lanes per block, 4 blocks at a time, one
// 16-byte store each -- a whole 128-byte line per block instead of one
// scattered 2-byte store per coefficient -- and clears those buffers.  Blocks
// go to memory whole, so the range needs no zero fill; a unit that stops at
// an error stores its partial block (as the serial decode leaves it).
// Measured on the 1024-image mix: 1.05 ms with a branch per event, tables in
// global memory and a store loop per symbol; 0.72 ms as here (48 1080p frames
// 0.35 -> 0.23, 512 thumbnails 0.25 -> 0.12).
template <bool GLOBAL>
static __device__ __noinline__ void cj_write_warp(CJWriteJob* job, bool active) {
  CJWriteJob& x = *job;
  const uint8_t* const set = x.gtab;
  const int lane = threadIdx.x & 31;
  cj_phase_entries(*x.sp, x.tab, x.phase);
  CJWin<CJ_WRITE_WORDS> br;
  const uint32_t mine = x.wbuf + 128 * lane, swz = (uint32_t)(lane & 7) << 4, zz = x.zz;
  // (copies: the compiler reads a job's fields from local memory again after
  // every shared-memory store of the loop)
  const uint32_t phases = x.phase, seg_end = x.marker ? x.seg_end : 0xFFFFFFFFu, order = x.order;
  const uint32_t wsrc = x.wbuf;
  uint4* const out = reinterpret_cast<uint4*>(x.coef) + (lane & 7);
  // a block does not start here by itself: the unit's or lane's end, or past the marker
  uint32_t lim = min(x.stop, x.last ? 0xFFFFFFFFu : x.end);
  lim = min(lim, seg_end);
  int b = x.blk, dc0 = x.dc[0], dc1 = x.dc[1], dc2 = x.dc[2];
  const int bend = x.bend;
  bool cut = false;
  uint32_t next = x.m;
  uint2 ph = make_uint2(cj_lds32(phases + 8 * next), cj_lds32(phases + 8 * next + 4));
  uint32_t tab, sh, ac1;
  int c, k = -1, dd = 0;
  auto begin_block = [&]() {
    tab = ph.x & 0xFFFFu;
    sh = 32 - CJ_MULTI_DC_BITS;
    ac1 = ph.y & 0xFFFFu;
    c = (int)((ph.y >> 16) & 255);
    next = ph.y >> 24;
    ph.x = cj_lds32(phases + 8 * next);
    ph.y = cj_lds32(phases + 8 * next + 4);
    k = -1;
  };
  // why no block starts at bit p (once per unit)
  auto stopped = [&](uint32_t p) {
    if (p >= x.stop || (!x.last && p >= x.end)) return;
    if (b >= bend) {
      if (!x.last) cj_raise_dec(x.st, x.base + b, CJ_DEV_EXTRA);
      // (where the last block ends; a unit that starts behind it starts where the speculative decode took
      // the padding bits for a block, and that may reach past the segment)
      else if (b == bend && (x.marker ? ((p + 7) >> 3) != x.end_byte : x.end_byte > ((p + 7) >> 3) + 2))
        cj_raise_dec(x.st, x.base + b, CJ_DEV_TRAILING);
    } else {
      cj_raise_dec(x.st, x.base + b, CJ_DEV_OVERRUN);
    }
  };
  br.pos = x.pos;
  br.col = x.ring;
  br.cur = br.nxt = br.nn = 0;
  bool live = active;
  if (live && (br.pos >= lim || b >= bend)) {
    stopped(br.pos);
    live = false;
  }
  if (live) br.init(x.data, x.ring, x.end_byte, br.pos);
  begin_block();
  if (!live) k = 63;
  uint32_t lst = 0;  // the block's last entry
  // One symbol of entry st at window v; DC only where `dc` says so.
  auto symbol = [&](uint32_t st, uint32_t v, bool dc) {
    const uint32_t size = (st >> 5) & 15, dk = st >> 9;
    const uint32_t w = __funnelshift_l(0u, v, (st & 31) - size);
    // (T.81 F.2.2.1: a magnitude whose first bit is 0 is negative)
    int val = (int)__funnelshift_rc(w, 0u, 32 - size);
    val -= (int)w >= 0 ? (int)((1u << size) - 1u) : 0;
    const bool isdc = dc && k < 0;
    if (dc) dd = isdc ? val : dd;
    br.skip(st & 31);
    k += (int)dk;
    if (size && dk - 1u < 16u && k <= 63 && !isdc) cj_sts16(mine + (cj_tab8(zz + k) ^ swz), (uint32_t)val);
    const bool prefix = dk == 0;
    tab = prefix ? ac1 + CJ_SPEC_SUB + ((st & 0x1E0u) << 2) : ac1;
    sh = prefix ? 26 : 32 - CJ_FAST_BITS;
  };
  while (__any_sync(CJ_FULL, live)) {
    if (live) br.refill();
    __syncwarp();
#pragma unroll
    for (int q = 0; q < CJ_STEPS_PER_ROUND; q++) {
      const uint32_t v = br.peek();
      uint32_t st = cj_entry<GLOBAL>(set, tab + 2 * (v >> sh));
      lst = k < 63 ? st : lst;
      st = k < 63 ? st : 0;
      symbol(st, v, q == 0);
    }
    bool done = false;
    if (live && k >= 63) {
      if (k >= CJ_SPEC_FARK) {  // rare: from the canonical table in memory
        k -= (int)(CJ_SPEC_FAR >> 9);
        const uint32_t v = br.peek();
        const uint32_t slot = k < 0 ? x.sp->comp_dc[c] : x.sp->comp_ac[c];
        lst = cj_spec_entry(cj_step_canonical(x.tp->huff[slot], slot, v), 0, k < 0);
        symbol(lst, v, true);
      }
      if (k >= 63) {
        done = true;
        const uint32_t adv = lst >> 9;
        // an EOB, or a symbol that landed on 63
        const bool ok = adv == CJ_SPEC_EOB ? (lst & 0x1E0u) == 0 : k == 63 && adv <= 16;
        if (!ok || br.pos > seg_end) {
          cj_raise_dec(x.st, x.base + b, ok ? CJ_DEV_OVERRUN : CJ_DEV_BAD_AC);
          cut = true;
        } else {
          int v = c == 0 ? dc0 : (c == 1 ? dc1 : dc2);
          v += dd;
          if (c == 0) dc0 = v;
          else if (c == 1) dc1 = v;
          else dc2 = v;
          if (v < -32768 || v > 32767) {
            cj_raise_dec(x.st, x.base + b, CJ_DEV_DC_RANGE);
            cut = true;
          } else {
            cj_sts16(mine + swz, (uint32_t)v);
          }
        }
      }
    }
    const unsigned mask = __ballot_sync(CJ_FULL, done);
    if (mask) {
      if (done) cj_sts_done(order + 8 * __popc(mask & ((1u << lane) - 1u)), cj_done(b, (uint32_t)lane));
      __syncwarp();
      const int n = __popc(mask);
      for (int r = lane >> 3; r < ((n + 3) & ~3); r += 4) {  // warp-uniform count
        if (r < n) {
          const CJDone o = cj_lds_done(order + 8 * r);
          const uint32_t at = wsrc + 128 * o.lane + ((((uint32_t)lane ^ o.lane) & 7u) << 4);
          const uint4 z = cj_lds128(at);
          out[cj_done_chunk(o)] = z;
          cj_sts128_zero(at);
        }
      }
      __syncwarp();
      if (done) {
        if (cut) {
          live = false;
        } else {
          b++;
          begin_block();
          if (br.pos >= lim || b >= bend) {
            stopped(br.pos);
            live = false;
          }
        }
        if (!live) k = 63;
      }
    }
  }
  x.blk = b;
  x.cut = cut;
}
