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
__device__ __forceinline__ void cj_sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Bit window of a lane in the warp-synchronous decode loops.  A lane's
// stream runs through a ring of CJ_RING_WORDS big-endian words in shared
// memory (word w in slot w mod CJ_RING_WORDS, `col` + 128 bytes per slot: one
// bank per lane, so every access is conflict-free at any progress of the
// lanes).  The current and the next word are in registers and the one after
// them is read a symbol ahead, without branches: a symbol's chain is a funnel
// shift, the table lookup, the position update and two selects.  Global memory
// is touched only in refill(), which the whole warp runs together once per
// CJ_RING_ROUNDS rounds of the loop: a 16-byte chunk fetched there has until
// the next refill to arrive.
// Bytes at or past `end_byte` read as 0xFF (the padding the reference's bit
// reader supplies); memory past them is not relied on.
#define CJ_RING_WORDS 16
#define CJ_STEPS_PER_ROUND 3
// rounds per refill: a round is three symbols of at most 31 bits, so three
// rounds cross at most 9 words; 9 + 2 read ahead + 3 of the oldest chunk < 16
#define CJ_RING_ROUNDS 3
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
    const uint32_t o = col + 128 * ((4 * c) & (CJ_RING_WORDS - 1));
#pragma unroll
    for (int i = 0; i < 4; i++) cj_sts32(o + 128 * i, w[i]);
  }
  // word pos / 32 + ahead
  __device__ __forceinline__ uint32_t word(uint32_t ahead) const {
    return cj_lds32(col + (((pos + 32 * ahead) << 2) & (128 * (CJ_RING_WORDS - 1))));
  }
  __device__ __forceinline__ void init(const uint4* data, uint32_t ring_col, uint32_t eb, uint32_t p) {
    chunks = data;
    col = ring_col;
    end_byte = eb;
    cb = p >> 7;
    uint4 v[CJ_RING_WORDS / 4];
#pragma unroll
    for (int i = 0; i < CJ_RING_WORDS / 4; i++) v[i] = load(cb + i);
    pf = load(cb + CJ_RING_WORDS / 4);
#pragma unroll
    for (int i = 0; i < CJ_RING_WORDS / 4; i++) put(cb + i, v[i]);
    pos = p;
    cur = word(0);
    nxt = word(1);
    nn = word(2);
  }
  // Replace the chunks the window has left behind.
  __device__ __forceinline__ void refill() {
    while ((pos >> 7) > cb) {
      put(cb + CJ_RING_WORDS / 4, pf);
      cb++;
      pf = load(cb + CJ_RING_WORDS / 4);
    }
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

// Bit reader of the decode loops: the current and the next big-endian word
// and a bit offset; a 32-bit window is one funnel shift, and a word boundary
// is crossed at most once per symbol (a symbol consumes at most 31 bits).
// One more word is loaded a crossing ahead and kept as read from memory
// (byte-swapped only when it becomes the next word), so a load has several
// symbols to arrive before the window needs it.
// Bytes at or past `end_byte` read as 0xFF (the padding the reference's bit
// reader supplies).
struct CJFBits {
  const uint32_t* words;
  uint32_t wfull, end_byte, cur, nxt, raw2, wi, off;

  __device__ __forceinline__ uint32_t word(uint32_t i) const {
    return i < wfull ? cj_bswap(words[i]) : cj_word(words, i, end_byte);
  }
  // word i as stored (cj_bswap of it is word(i))
  __device__ __forceinline__ uint32_t word_raw(uint32_t i) const {
    return i < wfull ? words[i] : cj_bswap(cj_word(words, i, end_byte));
  }
  __device__ __forceinline__ void init(const uint32_t* w, uint64_t eb, uint64_t p) {
    words = w;
    end_byte = (uint32_t)eb;
    wfull = (uint32_t)(eb >> 2);
    const uint32_t w0 = (uint32_t)(p >> 5);
    off = (uint32_t)(p & 31);
    cur = word(w0);
    wi = w0 + 1;
    nxt = word(wi);
    raw2 = word_raw(wi + 1);
  }
  __device__ __forceinline__ uint32_t peek() const { return __funnelshift_l(nxt, cur, off); }
  __device__ __forceinline__ void skip(uint32_t u) {
    off += u;
    if (off >= 32) {
      off -= 32;
      cur = nxt;
      nxt = cj_bswap(raw2);
      wi++;
      raw2 = word_raw(wi + 1);
    }
  }
  __device__ __forceinline__ uint64_t pos() const { return ((uint64_t)(wi - 1) << 5) + off; }
};

// Component, DC slot and AC slot of MCU phase m (from the packed phase
// table; the per-phase arrays for MCUs of more than 10 blocks).
__device__ __forceinline__ void cj_phase(const CJScanParams& sp, int bpm, uint64_t pack, uint32_t m, int& c,
                                         uint32_t& dslot, uint32_t& aslot) {
  if (bpm <= 10) {
    const uint32_t f = (uint32_t)(pack >> (6 * m)) & 63;
    c = (int)(f & 3);
    dslot = (f >> 2) & 3;
    aslot = f >> 4;
  } else {
    c = sp.phase_comp[m];
    dslot = sp.comp_dc[c];
    aslot = sp.comp_ac[c];
  }
}

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
// every step (measured: 870 cycles per symbol with branches for word
// crossings, long codes and block ends, against about 60 for the symbol's
// dependent instructions alone).  So word crossings are selects, a long code
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
// A warp's shared memory in the speculative decode: its ring, and per MCU
// phase the shared addresses of the phase's tables (x: dc | acm << 16), then
// ac1, the component << 16 and the next phase << 24 (y).
struct CJSpecWarp {
  uint32_t ring[CJ_RING_WORDS][32];
  uint2 phase[CJ_MAX_BPM];
};

// One lane's part of a decode: where and how (all lanes of the warp agree on
// sp, tp, tab), and its record in and out.
struct CJSpecJob {
  const CJScanParams *sp, *tp;
  const uint4* data;
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
                                            const CJSpecTab& tab, const void* data, const CJLane& ln, CJCkpt* ck,
                                            uint32_t cstep, const CJSpecWarp& sw) {
  x.sp = &sp;
  x.tp = &tp;
  x.tab = (uint32_t)__cvta_generic_to_shared(&tab);
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
template <bool HYP>
__device__ __noinline__ void cj_spec_warp(CJSpecJob* job, bool run, uint64_t start) {
  CJSpecJob& x = *job;
  CJWin br;
  const uint32_t begin = x.begin, end = x.end, cstep = x.cstep, phases = x.phase;
  CJCkpt* const ck = x.ck;
  const int bpm = x.sp->bpm;
  {  // the phase entries of this image and these tables
    const int i = threadIdx.x & 31;
    __syncwarp();
    if (i < bpm) {
      const uint32_t c = x.sp->phase_comp[i], d = x.sp->comp_dc[c], a = x.sp->comp_ac[c] - 2u;
      const uint32_t dc = x.tab + (uint32_t)offsetof(CJSpecTab, dc) + d * (uint32_t)sizeof(CJSpecTab::dc[0]);
      const uint32_t ac1 = x.tab + (uint32_t)offsetof(CJSpecTab, ac1) + a * (uint32_t)sizeof(CJSpecTab::ac1[0]);
      const uint32_t acm = x.tab + a * (uint32_t)sizeof(CJSpecTab::acm[0]);
      cj_sts32(phases + 8 * i, dc | (acm << 16));
      cj_sts32(phases + 8 * i + 4, ac1 | (c << 16) | ((i + 1 == bpm ? 0u : (uint32_t)i + 1) << 24));
    }
    __syncwarp();
  }
  static_assert(sizeof(CJSpecTab::sub[0]) == sizeof(CJSpecTab::ac1[0]), "sub follows ac1 at one distance");
  constexpr uint32_t SUB = (uint32_t)(offsetof(CJSpecTab, sub) - offsetof(CJSpecTab, ac1));
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
    tab = prefix ? ac1 + SUB + ((st & 0x1E0u) << 2) : (high ? ac1 : acm);
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
        uint32_t st = cj_tab16(tab + 2 * (v >> sh));
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
          const uint32_t st = cj_spec_entry(cj_step(*x.tp, k < 0 ? x.sp->comp_dc[c] : x.sp->comp_ac[c], v), 0, k < 0);
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
__device__ __forceinline__ bool cj_warp_settle(CJSpecJob& x, const CJLane& ln, uint64_t lane0_in) {
  int lane = threadIdx.x & 31;
  bool dirty = false;
  x.resume = true;
  for (int it = 0; it < 34; it++) {
    uint64_t pred = __shfl_up_sync(CJ_FULL, x.r.exit, 1);
    uint64_t want = ln.head ? x.r.start : (lane == 0 ? lane0_in : pred);
    bool change = ln.active && want != x.r.start;
    if (!__any_sync(CJ_FULL, change)) break;
    cj_spec_warp<false>(&x, change, want);
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

// Warp-cooperative write-out of 32 units (one per lane; `active` = false for
// lanes without one), symbol for symbol the serial block decode with the
// same structural checks.  Each lane builds its current block in its own
// 64-entry int16 buffer in shared memory (`wbuf` + lane * 64, all zero on
// entry and on return).  After every symbol the warp stores the blocks its
// lanes completed in that step: 8 lanes per block, 4 blocks per round, one
// 16-byte store each -- a whole 128-byte line per block instead of one
// scattered 2-byte store per coefficient -- and clears those buffers.  Blocks
// go to memory whole, so the range needs no zero fill; a unit that stops at
// an error stores its partial block (as the serial decode leaves it) and zeroes
// the rest of its range, up to `zero_end`.
__device__ __forceinline__ void cj_write_units_warp(const CJScanParams& sp, const CJScanParams& tp, const uint32_t* words,
                                                    const CJLane& ln, const CJSegment& seg, uint64_t start,
                                                    int64_t first_block, int dc0, int dc1, int dc2,
                                                    int16_t* __restrict__ coef, CJStatus* st, const uint8_t* zz,
                                                    uint64_t stop, int64_t zero_end, bool active, int16_t* wbuf) {
  const int lane = threadIdx.x & 31;
  int16_t* mine = wbuf + lane * 64;
  int64_t b = first_block;
  const int64_t bend = seg.first_block + seg.nblocks;
  const uint64_t seg_end = seg.bit_end;
  const int bpm = sp.bpm;
  const uint64_t pack = sp.phase_pack;
  CJFBits br;
  uint32_t m = 0, aslot = 0, slot = 0;
  int c = 0;
  if (active) {
    br.init(words, ln.end_byte, cj_state_bit(start));
    m = cj_state_phase(start);
    cj_phase(sp, bpm, pack, m, c, slot, aslot);
  }
  int k = -1;
  int32_t dd = 0;
  bool cut = false;  // stopped inside block b at an error
  // the structural checks made before every block; false = stop here
  auto block_start = [&]() -> bool {
    const uint64_t p = br.pos();
    if (p >= stop) return false;  // the next unit's first block
    if (!ln.last && p >= ln.end) return false;
    if (b >= bend) {
      if (!ln.last) cj_raise_dec(st, b, CJ_DEV_EXTRA);
      else if (seg.marker_follows) {
        if (((p + 7) >> 3) != ln.end_byte) cj_raise_dec(st, b, CJ_DEV_TRAILING);
      } else if (ln.end_byte > ((p + 7) >> 3) + 2) {
        cj_raise_dec(st, b, CJ_DEV_TRAILING);
      }
      return false;
    }
    if (seg.marker_follows && p >= seg_end) {
      cj_raise_dec(st, b, CJ_DEV_OVERRUN);
      return false;
    }
    return true;
  };
  bool run = active && block_start();
  for (;;) {
    int done = -1;  // block (of this image) to store after this step
    if (run) {
      const uint32_t v = br.peek();
      const uint32_t stp = cj_step(tp, slot, v);
      const uint32_t dk = (stp >> 5) & 127, size = stp >> 12, total = stp & 31;
      const int kn = k + (int)dk;
      const uint32_t len = total - size;
      const int32_t val = size ? cj_extend((v << len) >> (32 - size), size) : 0;
      if (k < 0) dd = val;
      else if (size && kn <= 63) mine[zz[kn]] = (int16_t)val;
      br.skip(total - (kn > 63 ? size : 0u));
      slot = aslot;
      if (kn < 63) {
        k = kn;
      } else if (kn > 63 && dk != CJ_STEP_EOB) {  // failing symbol: the block is cut here
        cj_raise_dec(st, b, dk == CJ_STEP_NO_CODE ? CJ_DEV_BAD_CODE : CJ_DEV_BAD_AC);
        done = (int)b;
        cut = true;
        run = false;
      } else if (seg.marker_follows && br.pos() > seg_end) {
        cj_raise_dec(st, b, CJ_DEV_OVERRUN);
        done = (int)b;
        cut = true;
        run = false;
      } else {
        int dcv;
        if (c == 0) dcv = dc0 += dd;
        else if (c == 1) dcv = dc1 += dd;
        else dcv = dc2 += dd;
        if (dcv < -32768 || dcv > 32767) {
          cj_raise_dec(st, b, CJ_DEV_DC_RANGE);
          cut = true;
          run = false;
        } else {
          mine[0] = (int16_t)dcv;
          b++;
          m = (m + 1 == (uint32_t)bpm) ? 0 : m + 1;
          cj_phase(sp, bpm, pack, m, c, slot, aslot);
          k = -1;
          run = block_start();
        }
        done = (int)(cut ? b : b - 1);
      }
    }
    unsigned mask = __ballot_sync(CJ_FULL, done >= 0);
    __syncwarp();
    while (mask) {  // warp-uniform: up to 4 blocks per round, lanes 8j..8j+7 take the j-th
      const int s0 = __ffs(mask) - 1;
      mask &= mask - 1;
      const int s1 = __ffs(mask) - 1;
      mask &= mask - 1;
      const int s2 = __ffs(mask) - 1;
      mask &= mask - 1;
      const int s3 = __ffs(mask) - 1;
      mask &= mask - 1;
      const int j = lane >> 3;
      const int src = j == 0 ? s0 : (j == 1 ? s1 : (j == 2 ? s2 : s3));
      const int bsrc = __shfl_sync(CJ_FULL, done, src < 0 ? 0 : src);
      if (src >= 0) {
        uint4* s = reinterpret_cast<uint4*>(wbuf + src * 64) + (lane & 7);
        reinterpret_cast<uint4*>(coef + (int64_t)bsrc * 64)[lane & 7] = *s;
        *s = make_uint4(0, 0, 0, 0);
      }
    }
    __syncwarp();
    if (!__any_sync(CJ_FULL, run)) break;
  }
  // blocks of the range an early stop left undecoded read as zeros
  for (int64_t x = cut ? b + 1 : b; active && x < zero_end; x++) {
    uint4* p = reinterpret_cast<uint4*>(coef + x * 64);
#pragma unroll
    for (int i = 0; i < 8; i++) p[i] = make_uint4(0, 0, 0, 0);
  }
}
