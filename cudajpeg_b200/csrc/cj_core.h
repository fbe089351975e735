// cj_core.h -- data layouts, Huffman tables and decode steps shared by the
// entropy kernels.  Everything here is plain C++ marked __host__ __device__
// so the same code is compiled for sm_100a kernels and for host checks of
// the table builder.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define CJ_HD __host__ __device__ __forceinline__
#else
#define CJ_HD inline
#endif

// ---------------------------------------------------------------- limits
#define CJ_FAST_BITS 10          // first-level Huffman lookup width
#define CJ_MAX_BPM 32            // blocks per MCU (the standard allows 10)
#define CJ_SUB_BITS_DEFAULT 1024 // bits per speculative subsequence
#define CJ_MAX_SCAN_BYTES (256u << 20) // block / bit counters are 32-bit

// Device error codes (the reader maps them to the format.h codes)
#define CJ_DEV_OK 0
#define CJ_DEV_BAD_CODE 1        // Huffman prefix with no code (SYNTAX_ERROR)
#define CJ_DEV_BAD_AC 2          // zero-size AC symbol that is not EOB/ZRL, or run past 63
#define CJ_DEV_OVERRUN 3         // restart interval needs bits past its marker
#define CJ_DEV_TRAILING 4        // restart interval has whole bytes after its last MCU
#define CJ_DEV_MARKER 5          // bad / missing / misplaced RSTn, or other marker in scan
#define CJ_DEV_DC_RANGE 6        // DC predictor outside int16 (UNSUPPORTED_ERROR)
#define CJ_DEV_EXTRA 7           // more entropy data than MCUs
#define CJ_DEV_CAPACITY 8        // more markers / subsequences than buffers allow
#define CJ_DEV_TIMEOUT 9         // a wait for another scan's blocks ran out (progressive.cu)

// One Huffman table in canonical form.
//   fast[w >> (16 - CJ_FAST_BITS)] = (len << 8) | symbol for codes of length
//   <= CJ_FAST_BITS, else 0; longer codes are found through maxcode/valoff
//   exactly as in ITU T.81 Annex F.2.2.3 (DECODE procedure).
struct CJHuff {
  uint16_t fast[1 << CJ_FAST_BITS];
  int32_t maxcode[18];  // [l], l = 1..16: largest code of length l, -1 if none
  int32_t valoff[18];   // symbol index of code c of length l = valoff[l] + c
  uint8_t vals[256];
};

// Decode steps: the per-symbol work of the entropy decoder, tabulated.
// Entry for a Huffman table slot and the next 10 bits of the stream:
//   bits 0-4   bits the symbol consumes: code length + magnitude size
//   bits 5-11  advance of the zig-zag position: DC 1 (from -1 to 0), AC
//              run + 1, ZRL 16, EOB 64, invalid AC symbol 96, no code 97
//   bits 12-15 magnitude size (extra bits that carry the value)
// An entry consuming 0 bits is a pointer: bits 5-15 index a 64-entry
// subtable for the following 6 bits (codes of 11-16 bits), or are
// CJ_STEP_SEARCH when the table has more long-code prefixes than subtables
// (the canonical search then decodes the code).  Long codes of a canonical
// table are the last codes of the code space, so their 10-bit prefixes form
// one contiguous range [pmin, pmax]: subtable i serves prefix pmin + i.
#define CJ_STEP_SUBS 16
#define CJ_STEP_SEARCH 0x7FFu
#define CJ_STEP_EOB 64u
#define CJ_STEP_BAD_AC 96u
#define CJ_STEP_NO_CODE 97u
#define CJ_STEP_BAD (1u | (CJ_STEP_NO_CODE << 5))  // consume 1 bit, end the block
struct CJSteps {
  uint16_t pri[4][1 << CJ_FAST_BITS];
  uint16_t sub[4][CJ_STEP_SUBS][64];
};

// Tables of the entropy loops, in shared memory.  One 16-bit entry:
//   bits 0-4   bits consumed (codes and magnitudes)
//   bits 5-8   one symbol: the magnitude size (15 for an invalid code, 0 for an
//              EOB); long code: its row in `sub`
//   bits 9-15  advance of the zig-zag position (DC 1, from -1 to 0; an EOB or an
//              invalid code adds 63, in a DC table 64); 0: the first 10 bits of
//              a longer code, decoded on from its row by the next 6 bits
// CJ_SPEC_FAR (nothing consumed, the position past every other): decode the
// symbol through the canonical table in memory -- DC codes of more than 9 bits and AC
// tables with more long-code prefixes than rows.
//   acm  (the speculative decode, which needs positions and DC sums but no AC
//        values) every whole symbol the next CJ_MULTI_BITS bits determine, as one entry,
//        while they advance by at most 16 together (an EOB after at most 15):
//        up to position CJ_MULTI_MAXK no symbol of an entry can lie behind the
//        block's end, so an entry is always taken whole
//   ac1  one symbol (positions above CJ_MULTI_MAXK, and the write-out)
// An 11-bit window holds 1.5 symbols on average at high bit rates and more
// than two at low ones.
#define CJ_MULTI_BITS 11
#define CJ_MULTI_DC_BITS 9
#define CJ_MULTI_MAXK 47
#define CJ_SPEC_FAR (127u << 9)
#define CJ_SPEC_FARK 126  // positions from here on: a CJ_SPEC_FAR entry (the rest end at 62 + 63)
#define CJ_SPEC_EOB 63u
struct CJSpecTab {
  uint16_t acm[2][1 << CJ_MULTI_BITS];
  uint16_t ac1[2][1 << CJ_FAST_BITS];
  uint16_t dc[2][1 << CJ_MULTI_DC_BITS];
  uint16_t sub[2][CJ_STEP_SUBS][64];
};

// Per-scan parameters, built on the host after SOS and copied once.
struct alignas(16) CJScanParams {
  CJHuff huff[4];                 // DC0, DC1, AC0, AC1
  int16_t qnat[4][64];            // quantisation tables, natural order
  uint8_t phase_comp[CJ_MAX_BPM]; // component of the k-th block of an MCU
  uint8_t phase_blk[CJ_MAX_BPM];  // index of that block inside its component's MCU part
  uint8_t comp_dc[3], comp_ac[3], comp_q[3];
  uint8_t comp_sx[3], comp_sy[3];
  uint8_t pad0;
  uint8_t zz[64];                 // natural-order index of zig-zag position k
  int32_t nch, bpm, mcux, mcuy;
  int32_t width, height;
  int32_t hmax, vmax, xshift, yshift; // chroma upsample shifts
  int32_t restart_interval;          // MCUs, 0 = none
  int32_t nseg_expected;             // restart intervals in the scan
  int64_t total_blocks;              // mcux*mcuy*bpm
  int32_t comp_stride[3];            // plane strides (bytes) for plane outputs
  int32_t comp_rows[3];
  int32_t tab;  // batch: the image whose decode tables serve this one (the same DHT contents)
};

// A restart interval (or the whole scan) in the destuffed buffer.
struct CJSegment {
  uint64_t bit_begin, bit_end;   // bits in the destuffed buffer
  int64_t first_block;           // global block index of its first block
  int64_t nblocks;               // blocks it must contain
  int32_t first_sub, nsub;       // its subsequences
  int32_t marker_follows;        // an RSTn ends it: its data must end on that
                                 // byte; otherwise reads past the end give 1-bits
  int32_t pad;
};

// A block completed by a lane of a write-out warp.  The block counts from the
// first block of the warp's first unit and takes a word of its own: another
// lane's unit may lie anywhere in the image before or behind it (the next
// restart interval begins at its own first block, however many blocks the data of
// the one before it holds, and a truncated scan's padding decodes to the image's end).
struct alignas(8) CJDone {
  int32_t block;
  uint32_t lane;
};
CJ_HD CJDone cj_done(int32_t block, uint32_t lane) { return CJDone{block, lane}; }
// Its first 16-byte chunk in the coefficient buffer, from the same origin.
CJ_HD int64_t cj_done_chunk(const CJDone& d) { return (int64_t)d.block * 8; }

// Positions of the write-out.  They are 32-bit and the data end at bit 2^31 at
// the latest (CJ_MAX_SCAN_BYTES), but the last unit of a truncated scan decodes
// on in 1-bits until its image's last block, which may take more than 2^32 of
// them.  A position this far behind the data and its chunk index are put back by
// whole rings of the bit window, to where there is still nothing but 1-bits.
#define CJ_POS_FOLD 0xC0000000u
#define CJ_POS_BACK (1u << 30)
CJ_HD void cj_fold_position(uint32_t& pos, uint32_t& chunk) {
  if (pos >= CJ_POS_FOLD) {
    pos -= CJ_POS_BACK;
    chunk -= CJ_POS_BACK / 128;
  }
}

// Decoder state at a block boundary: bit position and MCU phase.
CJ_HD uint64_t cj_state(uint64_t bit, uint32_t phase) { return (bit << 8) | phase; }
CJ_HD uint64_t cj_state_bit(uint64_t s) { return s >> 8; }
CJ_HD uint32_t cj_state_phase(uint64_t s) { return (uint32_t)(s & 0xFF); }

// One speculative subsequence: where its decode started, where it left off,
// how many blocks it began and the sum of its DC differences per component.
struct alignas(16) CJSubRec {
  uint64_t start;
  uint64_t exit;
  int32_t nblocks;
  int32_t dc[3];
};

// Per-warp aggregate used by the segmented block/DC scan.
struct alignas(16) CJWarpAgg {
  int32_t has_head;  // a segment starts inside this warp
  int32_t nblocks;   // sums over the lanes after the last segment head
  int32_t dc[3];
  int32_t pad[3];
};

// Status words the host reads back after a decode.
struct CJStatus {
  unsigned long long err_key;     // destuff / segment errors: complemented
                                  // min of (block << 8 | CJ_DEV_*), 0 = none
  unsigned long long dec_err_key; // errors of the coefficient write-out and
                                  // pixel passes (same encoding); cleared when
                                  // those passes are re-run
  int32_t unstable;           // warps whose last exit changed in the last fix-up pass
  int32_t nmarkers;           // RSTn markers found by the destuffer
  int32_t nsub;               // subsequences in use
  int32_t nseg;               // restart intervals in use
  int64_t destuffed;          // bytes after destuffing
};
#define CJ_NO_ERROR_KEY 0xFFFFFFFFFFFFFFFFull

// ---------------------------------------------------------------- bit access
CJ_HD uint32_t cj_bswap(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __byte_perm(v, 0, 0x0123);
#else
  return __builtin_bswap32(v);
#endif
}

// Decode one Huffman code from a left-aligned 16-bit window.  Returns
// (len << 8) | symbol, or 0 when no code of length 1..16 matches.
// Codes longer than CJ_FAST_BITS: canonical search by length.
CJ_HD uint32_t cj_huff_slow(const CJHuff& t, uint32_t win16) {
  for (int l = CJ_FAST_BITS + 1; l <= 16; l++) {
    int32_t code = (int32_t)(win16 >> (16 - l));
    if (code <= t.maxcode[l]) return ((uint32_t)l << 8) | t.vals[(t.valoff[l] + code) & 255];
  }
  return 0;
}

CJ_HD uint32_t cj_huff_decode(const CJHuff& t, uint32_t win16) {
  uint32_t e = t.fast[win16 >> (16 - CJ_FAST_BITS)];
  if (e) return e;
  return cj_huff_slow(t, win16);
}

// Decode step of a decoded (len << 8 | symbol) from a DC (ac = false) or AC table.
CJ_HD uint32_t cj_step_of(uint32_t e, bool ac) {
  if (!e) return CJ_STEP_BAD;
  const uint32_t len = e >> 8, sym = e & 255, size = sym & 15, run = sym >> 4;
  const uint32_t dk = !ac ? 1u : (size ? run + 1 : (sym == 0 ? CJ_STEP_EOB : (sym == 0xF0 ? 16u : CJ_STEP_BAD_AC)));
  return (len + size) | (dk << 5) | (size << 12);
}

// 10-bit prefixes of the codes longer than 10 bits, from the DHT counts
// (canonical assignment, T.81 Annex C); *pmin > *pmax when there are none.
CJ_HD void cj_long_prefixes(const uint8_t counts[16], int* pmin, int* pmax) {
  int code = 0;
  *pmin = 1 << CJ_FAST_BITS;
  *pmax = -1;
  for (int l = 1; l <= 16; l++) {
    const int n = counts[l - 1];
    if (l > CJ_FAST_BITS && n) {
      const int a = code >> (l - CJ_FAST_BITS), b = (code + n - 1) >> (l - CJ_FAST_BITS);
      if (a < *pmin) *pmin = a;
      if (b > *pmax) *pmax = b;
    }
    code = (code + n) << 1;
  }
}

// Primary step entry for prefix p of table t (its fast table already built).
CJ_HD uint16_t cj_step_primary(const CJHuff& t, int pmin, int pmax, int p, bool ac) {
  const uint32_t e = t.fast[p];
  if (e) return (uint16_t)cj_step_of(e, ac);
  if (p < pmin || p > pmax) return (uint16_t)CJ_STEP_BAD;
  const uint32_t i = (uint32_t)(p - pmin);
  return (uint16_t)((i < CJ_STEP_SUBS ? i : CJ_STEP_SEARCH) << 5);
}

// Entry j of subtable s (prefix pmin + s) of table t.
CJ_HD uint16_t cj_step_sub(const CJHuff& t, int pmin, int s, int j, bool ac) {
  const uint32_t win = ((uint32_t)(pmin + s) << 6) | (uint32_t)j;
  if (pmin + s >= (1 << CJ_FAST_BITS)) return (uint16_t)CJ_STEP_BAD;
  return (uint16_t)cj_step_of(cj_huff_slow(t, win), ac);
}

// The decode step for the 32-bit window v (MSB = next bit) from the step tables
// of `slot`; `t` is its canonical table.
CJ_HD uint32_t cj_step(const CJSteps& T, const CJHuff& t, uint32_t slot, uint32_t v) {
  uint32_t st = T.pri[slot][v >> (32 - CJ_FAST_BITS)];
  if (!(st & 31)) {
    const uint32_t i = st >> 5;
    st = i != CJ_STEP_SEARCH ? T.sub[slot][i][(v >> 16) & 63] : cj_step_of(cj_huff_slow(t, v >> 16), slot >= 2);
  }
  return st;
}
// The same step from the canonical table alone.
CJ_HD uint32_t cj_step_canonical(const CJHuff& t, uint32_t slot, uint32_t v) {
  return cj_step_of(cj_huff_decode(t, v >> 16), slot >= 2);
}

// Entries of the CJSpecTab from the decode steps: a step, a primary entry of an
// AC table, entry of a subtable.
CJ_HD uint16_t cj_spec_entry(uint32_t st, uint32_t behind, bool dc = false) {
  const uint32_t dk = (st >> 5) & 127, low = dk >= CJ_STEP_BAD_AC ? 15 : st >> 12;
  return (uint16_t)(((st & 31) - behind) | (low << 5) | ((dk >= CJ_STEP_EOB ? CJ_SPEC_EOB + dc : dk) << 9));
}
CJ_HD uint16_t cj_spec_ac1(uint32_t st) {
  if (st & 31) return cj_spec_entry(st, 0);
  return (st >> 5) == CJ_STEP_SEARCH ? (uint16_t)CJ_SPEC_FAR : (uint16_t)(CJ_FAST_BITS | ((st >> 5) << 5));
}
CJ_HD uint16_t cj_spec_sub(uint32_t st) {
  return cj_spec_entry(st, (st & 31) > CJ_FAST_BITS ? CJ_FAST_BITS : 0);  // (no code: 1 bit)
}
// The multi-symbol entry for the CJ_MULTI_BITS bits `idx` of an AC slot, from
// its primary step table.  Bits past the window read as 0 below, but a code
// after the first is taken only if it lies inside the window (its magnitude
// may reach past).
CJ_HD uint16_t cj_spec_acm(const uint16_t* pri, uint32_t idx) {
  const uint32_t v = idx << (32 - CJ_MULTI_BITS);
  uint32_t st = pri[v >> (32 - CJ_FAST_BITS)];
  if (!(st & 31) || ((st >> 5) & 127) > 16) return cj_spec_ac1(st);
  uint32_t used = st & 31, adv = (st >> 5) & 127;
  while (used < CJ_MULTI_BITS) {
    st = pri[(v << used) >> (32 - CJ_FAST_BITS)];
    const uint32_t total = st & 31, dk = (st >> 5) & 127, len = total - (st >> 12);
    if (!total || used + len > CJ_MULTI_BITS || used + total > 31) break;
    if (dk == CJ_STEP_EOB && adv <= 15) return (uint16_t)((used + total) | ((CJ_SPEC_EOB + adv) << 9));
    if (adv + dk > 16) break;
    used += total;
    adv += dk;
  }
  return (uint16_t)(used | (adv << 9));
}
// The entry for the CJ_MULTI_DC_BITS bits `idx` of a DC slot.
CJ_HD uint16_t cj_spec_dc(const uint16_t* pri, uint32_t idx) {
  const uint32_t st = pri[2 * idx];
  static_assert(CJ_FAST_BITS == CJ_MULTI_DC_BITS + 1, "two primary entries per DC entry");
  return (st & 31) && st == pri[2 * idx + 1] ? cj_spec_entry(st, 0, true) : (uint16_t)CJ_SPEC_FAR;
}

// Sign extension of a `size`-bit magnitude category value (T.81 F.2.2.1).
CJ_HD int32_t cj_extend(uint32_t bits, uint32_t size) {
  return (bits < (1u << (size - 1))) ? (int32_t)bits - (int32_t)(1u << size) + 1 : (int32_t)bits;
}

// Natural-order index of zig-zag position k (T.81 figure A.6).
#define CJ_ZIGZAG_INIT                                                                  \
  {0,  1,  8,  16, 9,  2,  3,  10, 17, 24, 32, 25, 18, 11, 4,  5,  12, 19, 26, 33, 40, 48, \
   41, 34, 27, 20, 13, 6,  7,  14, 21, 28, 35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, \
   30, 37, 44, 51, 58, 59, 52, 45, 38, 31, 39, 46, 53, 60, 61, 54, 47, 55, 62, 63}
