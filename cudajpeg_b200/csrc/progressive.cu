// progressive.cu -- progressive JPEG (SOF2) scans on the GPU.
//
// The reference decodes baseline frames only: SOF2 falls to its marker
// switch's SYNTAX_ERROR (src/format.cu:191-200).  Here a progressive frame
// goes through the same marker loop: every SOS (decodeScanGPU) is checked and
// noted, and the EOI's pixel stage first decodes the noted scans into the int16
// coefficient blocks (quantised, natural order, MCU scan order -- the layout of
// a baseline scan).  Scan types follow ITU T.81 Annex G (G.1.2): DC first
// (interleaved or not), DC refinement (one bit per block), AC first with
// end-of-band runs, and AC refinement with correction bits.
//
// One CTA per restart interval of a scan (a thread per interval, and a launch per scan,
// where the intervals are many and short).  A scan that touches coefficients of
// scans before it follows them: all scans run in one launch, and a chunk of
// blocks is decoded once the scans it follows have published that they are past
// these blocks (the refinements of a component run a chunk behind one another).
// If there are more intervals than CTAs fit on the GPU at once, a launch takes one
// level of scans, those whose predecessors all ran in the launches before.
// Noted scans take memory (some 10 KB each, for as little as ten bytes of file), so
// a frame's are decoded whenever PG_NOTE_SCANS of them, or PG_NOTE_INTERVALS
// intervals, have been noted; the usual script of ten scans never gets there.
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "../../include/decodeScanGPU.h"
#include "cj_entropy.cuh"
#include "cj_internal.h"
#include "cj_tables.h"

#define PG_NOTE_SCANS 64
#define PG_NOTE_INTERVALS (1u << 16)
#define PG_DEPS 16  // scans that one scan follows (64 bands at the most; more take the launch per level)

// A scan and its four Huffman tables.
struct CJProgTables {
  CJProgScan s;
  CJHuff huff[4];
};

// A scan's parameter block: with them the scans it follows in the same launch (block
// by block, or after their last: whole).
struct CJProgBlock : CJProgTables {
  int32_t ndep, dep[PG_DEPS];
  uint32_t whole;  // bit per dependency
  int32_t blocks;  // of the scan in all
};

// One CTA's work: a restart interval of a scan, its stuffed bytes [begin, end).
struct CJProgWork {
  int64_t begin, end;
  int32_t scan, iv;
};

// One CTA decodes one interval in chunks.  What is serial in such a scan is the
// walk from symbol to symbol: where a symbol lies depends on all before it,
// in a refinement scan on the block's history too, so no decode from the
// middle falls into step.  Everything else is taken out of that walk and done
// by all threads: before it, the chunk's bytes are destuffed, the symbol at
// EVERY bit position is decoded (sym), and for a refinement scan the
// zero-history positions of every block are listed (zpos); after it, the
// coefficients of the symbols found (evt) are read and written.  The walk itself,
// one thread, is then two dependent shared-memory loads per refinement symbol and
// one per symbol otherwise.
// Measured on a 1024x768 4:2:0 q80 file of 115 KB, 213 thousand symbols: 254 ms with
// one thread decoding each scan from global memory; in chunks, a launch per level
// of scans 17.4 ms with a walk of 132 cycles a symbol, 13.1 ms with the present one
// (1.5 + 3.8 + 7.6, the last luma refinement's 129 thousand symbols); in one launch
// 8.1 ms; with a refinement's blocks staged in shared memory 7.6 ms, and with no more in
// its walk than the next position takes 6.7 ms (about 95 cycles a symbol in all; loading
// the four nearest entries ahead, to save the second load's latency, 9.3 ms: the
// instructions count too).
#define PG_THREADS 512
#define PG_BITS 16384        // bit positions of a chunk
#define PG_BLOCK_BITS 2048   // no block takes more bits than this (63 symbols of 31 bits and an EOB)
#define PG_BYTES (PG_BITS / 8 + 16)
#define PG_SEQ 2048          // blocks of a chunk (first scans)
#define PG_REF_BLOCKS 256    // blocks of a chunk (AC refinement)
#define PG_EVENTS 4096
#define PG_ZPOS 128          // 63 positions, and the 64 a symbol may step behind them
#define PG_ZEND 252          // behind a block's last zero-history position
#define PG_RAW 9             // stuffed bytes a thread looks at per chunk

struct PGShared {
  CJHuff huff[2];                       // DC: slots 0 and 1; AC: [0]
  alignas(16) uint32_t ahead[64];       // the refinement walk may load up to 63 entries before sym (and not use them)
  union {
    alignas(16) uint32_t sym[PG_BITS];      // AC scans
    alignas(16) uint16_t dcsym[2][PG_BITS];  // DC scans: by Huffman table
  };
  alignas(16) uint8_t zpos[PG_REF_BLOCKS][PG_ZPOS];  // 4 x the zero-history positions of each block, then PG_ZEND
  alignas(16) uint32_t words[PG_BYTES / 4 + 4];  // destuffed bytes as stored, zeros behind them
  uint16_t raw[PG_BYTES + 1];           // offset of each destuffed byte from the chunk's first stuffed byte
  uint32_t evt[PG_EVENTS];
  uint32_t ev0[PG_SEQ];
  uint32_t coef[PG_REF_BLOCKS][33];     // the blocks before the scan (33: a thread per block, each in a bank of its own)
  uint64_t hist[PG_REF_BLOCKS];         // nonzero coefficients of the band, bit = zig-zag position - ss
  uint8_t nz[PG_REF_BLOCKS + 1];
  uint8_t zz[64];
  uint8_t pcomp[CJ_MAX_BPM], pslot[CJ_MAX_BPM];
  int32_t pofs[CJ_MAX_BPM];
  int2 scan[33];
  // the walk's state between chunks
  int64_t rawpos;
  int bit, blk, eob, err, dc[3];
  int pos, done;  // after the walk: bits and blocks of this chunk
  int ready;      // the scans before it are past this chunk's blocks
  int range;      // its first block with a value outside int16 (INT_MAX: none)
};

// Symbol entries.  DC (16 bits): bits 0-4 bits consumed, 5-8 magnitude size, 15
// invalid.  AC (32 bits): byte 0 four times the bits consumed (sym's bytes to the
// next entry); byte 1 run + 1, or PG_STEP_OUT, which leaves the band, for an
// end-of-band run (PG_EOB; bits 16-30: the further blocks it covers; its extra
// bits count as consumed) and for an invalid code (PG_BAD); byte 2 first scans:
// magnitude size, refinement: 1 newly nonzero, 3 and negative.  (ZRL is a run of
// 15 with byte 2 zero.)
#define PG_DC_BAD 0x8000u
#define PG_EOB 0x80000000u
#define PG_BAD 0x40000000u
#define PG_STEP_OUT 64u
__device__ __forceinline__ uint32_t pg_dc_symbol(const CJHuff& t, uint32_t win) {
  const uint32_t e = cj_huff_decode(t, win >> 16), s = e & 255;
  return !e || s > 11 ? PG_DC_BAD : ((e >> 8) + s) | (s << 5);
}
__device__ __forceinline__ uint32_t pg_ac_symbol(const CJHuff& t, uint32_t win, bool refine) {
  const uint32_t e = cj_huff_decode(t, win >> 16);
  const uint32_t len = e >> 8, r = (e >> 4) & 15, s = e & 15;
  if (!e || (refine && s > 1)) return PG_BAD | (PG_STEP_OUT << 8);
  if (s == 0 && r < 15) {
    const uint32_t more = (1u << r) - 1u + __funnelshift_rc(win << len, 0u, 32 - r);
    return (4 * (len + r)) | (PG_STEP_OUT << 8) | (more << 16) | PG_EOB;
  }
  const uint32_t low = (4 * (len + s)) | ((r + 1) << 8);
  if (!refine) return low | (s << 16);
  return low | (s ? ((win >> (31 - len)) & 1u ? 1u : 3u) << 16 : 0u);
}

// 32 bits of the chunk from bit p on.
__device__ __forceinline__ uint32_t pg_peek(const PGShared& S, uint32_t p) {
  const uint32_t w = p >> 5;
  return __funnelshift_l(cj_bswap(S.words[w + 1]), cj_bswap(S.words[w]), p);
}
__device__ __forceinline__ uint32_t pg_bits(const PGShared& S, uint32_t p, uint32_t n) {
  return __funnelshift_rc(pg_peek(S, p), 0u, 32 - n);
}

// Block of the coefficient buffer that is the i-th of the interval.
__device__ __forceinline__ int64_t pg_block(const CJProgScan& s, const PGShared& S, int u0, int bps, int i) {
  if (s.ns > 1) {
    const int u = i / bps;
    return (int64_t)(u0 + u) * s.bpm + S.pofs[i - u * bps];
  }
  const int u = u0 + i, bx = u % s.bw, by = u / s.bw;
  const int64_t mcu = (int64_t)(by / s.sy[0]) * s.mcux + bx / s.sx[0];
  return mcu * s.bpm + s.first[0] + (by % s.sy[0]) * s.sx[0] + bx % s.sx[0];
}

// The chunk's bytes, destuffed (a zero byte after FF is dropped).
__device__ __forceinline__ void pg_stage_bytes(PGShared& S, const uint8_t* __restrict__ file, int64_t begin, int64_t end) {
  const int t = threadIdx.x;
  uint32_t b[PG_RAW + 1];
  const int64_t at = begin + (int64_t)t * PG_RAW;
  b[0] = t && at - 1 < end ? file[at - 1] : 0;  // (the byte before the chunk is not an FF with a zero behind it)
#pragma unroll
  for (int j = 0; j < PG_RAW; j++) b[j + 1] = at + j < end ? file[at + j] : 0x100;
  int n = 0;
#pragma unroll
  for (int j = 1; j <= PG_RAW; j++) n += b[j] < 0x100 && !(b[j] == 0 && b[j - 1] == 0xFF);
  int2 tot;
  int o = cj_block_exclusive(make_int2(n, 0), S.scan, &tot).x;
  uint8_t* bytes = reinterpret_cast<uint8_t*>(S.words);
#pragma unroll
  for (int j = 1; j <= PG_RAW; j++)
    if (b[j] < 0x100 && !(b[j] == 0 && b[j - 1] == 0xFF)) {
      if (o < PG_BYTES) {
        bytes[o] = (uint8_t)b[j];
        S.raw[o] = (uint16_t)(t * PG_RAW + j - 1);
      }
      o++;
    }
  const int kept = min(tot.x, PG_BYTES);
  for (int k = kept + t; k < (int)sizeof(S.words); k += PG_THREADS) bytes[k] = 0;
  // behind the last byte of the interval the stream goes on as zeros
  for (int k = kept + t; k <= PG_BYTES; k += PG_THREADS) S.raw[k] = (uint16_t)min((int64_t)65535, end - begin);
  S.done = kept * 8;  // (every thread the same value) bits staged
  __syncthreads();
}
static_assert(PG_THREADS * PG_RAW >= 2 * PG_BYTES, "every second byte may be dropped");

// The symbol at every bit position of the chunk, 8 positions per thread and
// step (positions behind the data decode zeros).
template <bool DC>
__device__ __forceinline__ void pg_stage_symbols(PGShared& S, int which, const CJHuff& t, bool refine, int nbits) {
  const uint32_t zero = DC ? pg_dc_symbol(t, 0u) * 0x10001u : pg_ac_symbol(t, 0u, refine);
  for (int p = threadIdx.x * 8; p < PG_BITS; p += PG_THREADS * 8) {
    uint32_t out[8];
    if (p < nbits) {
      const uint32_t w0 = pg_peek(S, p), w1 = pg_peek(S, p + 8);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        // 32 bits from p + j: from w0 and the bits 8 .. 39 behind p
        const uint32_t win = j ? (w0 << j) | ((w1 << 24) >> (32 - j)) : w0;
        out[j] = DC ? pg_dc_symbol(t, win) : pg_ac_symbol(t, win, refine);
      }
      if (DC) {
#pragma unroll
        for (int j = 0; j < 4; j++) out[j] = out[2 * j] | (out[2 * j + 1] << 16);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) out[j] = zero;
    }
    if (DC) {
      *reinterpret_cast<uint4*>(&S.dcsym[which][p]) = make_uint4(out[0], out[1], out[2], out[3]);
    } else {
      reinterpret_cast<uint4*>(&S.sym[p])[0] = make_uint4(out[0], out[1], out[2], out[3]);
      reinterpret_cast<uint4*>(&S.sym[p])[1] = make_uint4(out[4], out[5], out[6], out[7]);
    }
  }
}

// ---- the walks (one thread).  Each stops before a block that might not fit
// the chunk and leaves S.pos, S.done (blocks), S.eob, S.err.

__device__ __forceinline__ void pg_walk_dc(PGShared& S, int nb, int bps) {
  uint32_t pos = S.bit;
  int b = 0, ph = S.blk % bps;
  for (; b < nb && pos < PG_BITS - PG_BLOCK_BITS; b++) {
    const uint32_t e = S.dcsym[S.pslot[ph]][pos];
    if (e & PG_DC_BAD) {
      S.err = CJ_DEV_BAD_AC;
      break;
    }
    const uint32_t size = (e >> 5) & 15;
    pos += e & 31;
    S.ev0[b] = (pos - size) | (size << 16);
    ph = ph + 1 == bps ? 0 : ph + 1;
  }
  S.pos = (int)pos;
  S.done = b;
}

// The AC walks keep positions as byte offsets into sym (four times the bit), load
// the next entry before they test whether the block ends, and leave the band by
// the same test at its last coefficient, an end-of-band run and an invalid code.
__device__ __forceinline__ uint32_t pg_lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t pg_lds8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}

// Event: offset of a symbol, its zig-zag position << 16.
__device__ __forceinline__ void pg_walk_first(PGShared& S, int nb, int ss, int se) {
  const uint32_t sym = (uint32_t)__cvta_generic_to_shared(S.sym);
  uint32_t pos = 4 * S.bit, e = pg_lds32(sym + pos);
  int b = 0, eob = S.eob, ne = 0;
  for (;;) {
    if (eob) {
      const int skip = min(eob, nb - b);
      b += skip;
      eob -= skip;
    }
    if (b >= nb || pos >= 4 * (PG_BITS - PG_BLOCK_BITS) || ne >= PG_EVENTS - 64) break;
    const int st = ne;
    int k = ss - 1;
    for (;;) {
      k += (int)((e >> 8) & 255);
      S.evt[ne++] = pos | ((uint32_t)k << 16);
      pos += e & 255;
      const uint32_t next = pg_lds32(sym + pos);
      if (k >= se) {
        if (k > se) {  // an end-of-band run, an invalid code, a coefficient past the band, a ZRL that ends the block
          ne--;
          if (e & PG_EOB) eob = (int)((e >> 16) & 0x7FFF);
          else if (e & PG_BAD) S.err = CJ_DEV_BAD_CODE;
          else if (e & 0xFF0000u) S.err = CJ_DEV_BAD_AC;
        }
        e = next;
        break;
      }
      e = next;
    }
    S.ev0[b] = (uint32_t)st | ((uint32_t)(ne - st) << 16);
    if (S.err) break;
    b++;
  }
  S.pos = (int)(pos >> 2);
  S.done = b;
  S.eob = eob;
}

// Refinement.  After a symbol with run r the block stands behind its (z + r)-th
// zero-history coefficient (z so far), at zig-zag position k = zpos[z + r], and
// has met k - (z + r) nonzero ones, whose correction bits lie behind the
// symbols: with q the bits of the block's symbols alone, the next symbol is at
// q + k - (z + r).  Every block takes one correction bit per nonzero coefficient
// in all.  Event: shared address of a symbol's entry; PG_IN_RUN: a block inside a run,
// of its correction bits (by position).
// One thread issues an instruction every 4 cycles or so: what the loop does not need
// (z + r, the band position) is left to those who read the events.
#define PG_IN_RUN 0x80000000u
__device__ __forceinline__ void pg_walk_refine(PGShared& S, int nb, int width) {
  const uint32_t sym = (uint32_t)__cvta_generic_to_shared(S.sym), zpos = (uint32_t)__cvta_generic_to_shared(S.zpos);
  const uint32_t last = 4 * (uint32_t)(width - 1), stop = sym + 4 * (PG_BITS - PG_BLOCK_BITS);
  uint32_t pos = sym + 4 * S.bit, e = pg_lds32(pos), nz_next = 4u * S.nz[0];
  int b = 0, eob = S.eob;
  uint32_t* evt = S.evt;
  while (b < nb && pos < stop && evt < S.evt + PG_EVENTS - 64) {
    const uint32_t nz4 = nz_next;
    nz_next = 4u * S.nz[b + 1];
    S.ev0[b] = (uint32_t)(evt - S.evt);
    if (eob) {
      *evt++ = pos | PG_IN_RUN;
      pos += nz4;
      e = pg_lds32(pos);
      eob--;
      b++;
      continue;
    }
    const uint32_t z0 = zpos + b * PG_ZPOS;
    uint32_t q = pos + 4, z = z0 - 1, k4, next;  // q: behind the block's symbols alone, less 4 (z + r); z + r = -1
    for (;;) {
      const uint32_t run = (e >> 8) & 255;
      z += run;
      k4 = pg_lds8(z);
      q = q + (e & 255) - 4 * run;
      *evt++ = pos;
      const uint32_t at = q + k4;
      next = pg_lds32(at);
      if (k4 >= last) {
        if (k4 < PG_ZEND) {
          pos = at;
          e = next;
        }
        break;
      }
      pos = at;
      e = next;
    }
    if (k4 >= PG_ZEND) {  // past the band: an end-of-band run, an error, or a ZRL that ends the block
      pos = q + 4 * (z - z0) + nz4;
      next = pg_lds32(pos);
      if (e & PG_EOB) {
        eob = (int)((e >> 16) & 0x7FFF);
      } else if (e & (PG_BAD | 0xFF0000u)) {
        S.err = CJ_DEV_BAD_AC;
        break;
      }
      e = next;
    }
    b++;
  }
  S.pos = (int)((pos - sym) >> 2);
  S.done = b;
  S.eob = eob;
  if (!S.err) S.ev0[b] = (uint32_t)(evt - S.evt);  // the end of the last block's events (an error's block is left out)
}

__constant__ uint8_t c_prog_zz[64] = CJ_ZIGZAG_INIT;

// Waits (one thread) until the scans that `b` follows are past `need` blocks of
// theirs, which of a dependency marked whole are all.  progress[i]: blocks of scan i
// done and written, progress[nscans]: chunks done by any CTA.  The wait is given up
// when no CTA of the launch finished a chunk for `limit` polls (by default seconds; a
// chunk takes a fraction of a millisecond, and the CTAs are all resident).
// Polls are relaxed loads, which leave the SM's L1 alone; the fence behind them
// orders the reads of the coefficients.
#define PG_WAIT_POLLS (1u << 23)
__device__ __forceinline__ int pg_load_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __noinline__ bool pg_await(const CJProgBlock* __restrict__ scans, const CJProgBlock& b, const int* progress,
                                      int nscans, int need, unsigned limit) {
  for (int j = 0; j < b.ndep; j++) {
    const int want = (b.whole >> j) & 1 ? scans[b.dep[j]].blocks : need;
    int seen = -1;
    unsigned polls = 0;
    while (pg_load_relaxed(&progress[b.dep[j]]) < want) {
      const int any = pg_load_relaxed(&progress[nscans]);
      if (any != seen) polls = 0;
      seen = any;
      if (++polls >= limit) return false;
      __nanosleep(256);
    }
  }
  __threadfence();
  return true;
}
// A CTA's chunk is written (its threads are past a barrier): blocks more of `scan` done.
__device__ __forceinline__ void pg_publish(int* progress, int nscans, int scan, int blocks) {
  __threadfence();
  atomicAdd(&progress[scan], blocks);
  atomicAdd(&progress[nscans], 1);
}

__global__ void __launch_bounds__(PG_THREADS) k_prog_scans(const CJProgBlock* __restrict__ scans,
                                                           const CJProgWork* __restrict__ work,
                                                           const uint8_t* __restrict__ file, int16_t* coef,
                                                           CJStatus* st, int* progress, int nscans,
                                                           unsigned wait_limit) {
  extern __shared__ __align__(16) uint8_t pg_smem[];
  PGShared& S = *reinterpret_cast<PGShared*>(pg_smem);
  const CJProgWork wk = work[blockIdx.x];
  const CJProgScan& s = scans[wk.scan].s;
  const int tid = threadIdx.x;
  const bool dc = s.ss == 0, refine = s.ah != 0;
  const int al = s.al, width = s.se - s.ss + 1;
  int bps = 1;
  if (s.ns > 1) {
    bps = 0;
    for (int j = 0; j < s.ns; j++) bps += s.sx[j] * s.sy[j];
  }
  for (int h = 0; h < 2; h++) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&scans[wk.scan].huff[dc ? h : s.ac_slot[0]]);
    for (int k = tid; k < (int)(sizeof(CJHuff) / 4); k += PG_THREADS) reinterpret_cast<uint32_t*>(&S.huff[h])[k] = src[k];
  }
  if (tid < 64) S.zz[tid] = c_prog_zz[tid];
  if (tid == 0) {
    for (int j = 0, k = 0; j < s.ns; j++)
      for (int w = 0; w < (s.ns > 1 ? s.sx[j] * s.sy[j] : 1); w++, k++) {
        S.pcomp[k] = (uint8_t)j;
        S.pslot[k] = (uint8_t)(s.dc_slot[j] & 1);
        S.pofs[k] = s.first[j] + w;
      }
    S.rawpos = wk.begin;
    S.bit = S.blk = S.eob = S.err = 0;
    S.range = INT_MAX;
    S.dc[0] = S.dc[1] = S.dc[2] = 0;
  }
  const int u0 = s.ri ? wk.iv * s.ri : 0;
  const int u1 = s.ri ? min(s.nunits, u0 + s.ri) : s.nunits;
  const int nseq = (u1 - u0) * bps;
  __syncthreads();
  while (S.blk < nseq && !S.err) {  // CTA-uniform: written only between barriers below
    const int blk0 = S.blk;
    const int64_t raw0 = S.rawpos;
    if (progress && scans[wk.scan].ndep) {
      // (a word of its own: S.err, which the loop's test reads, does not change before the next barrier)
      if (tid == 0)
        S.ready = pg_await(scans, scans[wk.scan], progress, nscans, min(nseq, blk0 + PG_REF_BLOCKS), wait_limit);
      __syncthreads();
      if (!S.ready) {
        if (tid == 0) cj_raise(st, 0, CJ_DEV_TIMEOUT);
        break;
      }
    }
    pg_stage_bytes(S, file, raw0, wk.end);
    const int nbits = S.done;
    int nb = nseq - blk0;
    if (dc && refine) {  // one bit per block, no walk
      nb = min(nb, PG_BITS - 8);
      const int bit0 = S.bit;
      for (int i = tid; i < nb; i += PG_THREADS)
        if (pg_bits(S, bit0 + i, 1)) {
          int16_t* c = coef + pg_block(s, S, u0, bps, blk0 + i) * 64;
          *c = (int16_t)(*c | (1 << al));
        }
      __syncthreads();
      if (tid == 0) {
        S.pos = bit0 + nb;
        S.done = nb;
      }
    } else {
      nb = min(nb, !dc && refine ? PG_REF_BLOCKS : PG_SEQ);
      if (dc) {
        pg_stage_symbols<true>(S, 0, S.huff[0], false, nbits);
        pg_stage_symbols<true>(S, 1, S.huff[1], false, nbits);
      } else {
        pg_stage_symbols<false>(S, 0, S.huff[0], refine, nbits);
      }
      if (dc) {
      } else if (refine) {  // the blocks, then their history: a warp per block, two zig-zag positions per lane
        const int lane = tid & 31;
        for (int i = tid; i < nb * 8; i += PG_THREADS) {
          const uint4 v = reinterpret_cast<const uint4*>(coef + pg_block(s, S, u0, bps, blk0 + (i >> 3)) * 64)[i & 7];
          uint32_t* to = &S.coef[i >> 3][4 * (i & 7)];
          to[0] = v.x;
          to[1] = v.y;
          to[2] = v.z;
          to[3] = v.w;
        }
        __syncthreads();
        const uint32_t lt = (1u << lane) - 1u;
        for (int b = tid >> 5; b < nb; b += PG_THREADS / 32) {
          const int16_t* blk = reinterpret_cast<const int16_t*>(S.coef[b]);
          const bool in0 = lane < width, in1 = lane + 32 < width;
          const bool n0 = in0 && blk[S.zz[s.ss + lane]] != 0, n1 = in1 && blk[S.zz[min(63, s.ss + lane + 32)]] != 0;
          const uint32_t h0 = __ballot_sync(CJ_FULL, n0), h1 = __ballot_sync(CJ_FULL, n1);
          const uint32_t z0 = __ballot_sync(CJ_FULL, in0 && !n0), z1 = __ballot_sync(CJ_FULL, in1 && !n1);
          if (lane < PG_ZPOS / 4) reinterpret_cast<uint32_t*>(S.zpos[b])[lane] = PG_ZEND * 0x01010101u;
          __syncwarp();
          if (in0 && !n0) S.zpos[b][__popc(z0 & lt)] = (uint8_t)(4 * lane);
          if (in1 && !n1) S.zpos[b][__popc(z0) + __popc(z1 & lt)] = (uint8_t)(4 * (lane + 32));
          if (lane == 0) {
            S.nz[b] = (uint8_t)(__popc(h0) + __popc(h1));
            S.hist[b] = (uint64_t)h0 | ((uint64_t)h1 << 32);
          }
        }
      } else {
        for (int b = tid; b < nb; b += PG_THREADS) S.ev0[b] = 0;
      }
      __syncthreads();
      if (tid == 0) {
        if (dc) pg_walk_dc(S, nb, bps);
        else if (refine) pg_walk_refine(S, nb, width);
        else pg_walk_first(S, nb, s.ss, s.se);
      }
      __syncthreads();
      const int done = S.done;
      if (dc) {  // differences, then a running sum per component (a warp each), then the coefficients
        int* val = reinterpret_cast<int*>(S.evt);
        for (int b = tid; b < done; b += PG_THREADS) {
          const uint32_t e = S.ev0[b], size = e >> 16;
          val[b] = size ? cj_extend(pg_bits(S, e & 0xFFFFu, size), size) : 0;
        }
        __syncthreads();
        if (tid < 32 * s.ns) {
          const int c = tid >> 5, lane = tid & 31;
          int run = S.dc[c];
          for (int b0 = 0; b0 < done; b0 += 32) {
            const int b = b0 + lane;
            const bool mine = b < done && S.pcomp[(blk0 + b) % bps] == c;
            int v = mine ? val[b] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
              const int o = __shfl_up_sync(CJ_FULL, v, d);
              if (lane >= d) v += o;
            }
            if (mine) S.ev0[b] = (uint32_t)(run + v);
            run += __shfl_sync(CJ_FULL, v, 31);
          }
          if (lane == 0) S.dc[c] = run;
        }
        __syncthreads();
        for (int b = tid; b < done; b += PG_THREADS) {
          const int64_t at = pg_block(s, S, u0, bps, blk0 + b);
          const int64_t v = (int64_t)(int)S.ev0[b] * (1 << al);
          if (v < -32768 || v > 32767) atomicMin(&S.range, b);
          else coef[at * 64] = (int16_t)v;
        }
      } else if (!refine) {
        const int last = min(nb, done + (S.err ? 1 : 0));  // with what precedes an error in its block
        for (int b = tid; b < last; b += PG_THREADS) {
          const uint32_t v0 = S.ev0[b];
          if (!(v0 >> 16)) continue;
          int16_t* blk = coef + pg_block(s, S, u0, bps, blk0 + b) * 64;
          for (uint32_t i = 0; i < (v0 >> 16); i++) {
            const uint32_t ev = S.evt[(v0 & 0xFFFFu) + i], e = S.sym[(ev & 0xFFFFu) >> 2], size = (e >> 16) & 255;
            if (!size) continue;  // ZRL
            const int v = cj_extend(pg_bits(S, (((ev & 0xFFFFu) + (e & 255)) >> 2) - size, size), size) * (1 << al);
            if (v < -32768 || v > 32767) {
              atomicMin(&S.range, b);
              break;
            }
            blk[S.zz[ev >> 16]] = (int16_t)v;
          }
        }
      } else {
        const int p1 = 1 << al, m1 = -(1 << al);
        const uint32_t sym = (uint32_t)__cvta_generic_to_shared(S.sym);
        for (int b = tid; b < done; b += PG_THREADS) {
          int16_t* blk = coef + pg_block(s, S, u0, bps, blk0 + b) * 64;
          uint64_t h = S.hist[b];
          const int nz = S.nz[b];
          const int e1 = (int)S.ev0[b + 1];
          int c = 0;          // corrections made
          uint32_t z = ~0u;  // zero-history coefficients passed, less 1
          for (int i = (int)S.ev0[b]; i < e1; i++) {
            const uint32_t ev = S.evt[i], off = (ev & ~PG_IN_RUN) - sym, e = S.sym[off >> 2];
            const bool in_run = (ev & PG_IN_RUN) != 0;
            z += (e >> 8) & 255;
            const uint32_t k4 = in_run ? PG_ZEND : S.zpos[b][z], k = k4 >> 2;
            const int c1 = k4 < PG_ZEND ? (int)(k - z) : nz;
            uint32_t at = (off + (in_run ? 0u : e & 255)) >> 2;
            for (; c < c1; c++, at++) {
              const int zz = S.zz[s.ss + __ffsll((long long)h) - 1];
              const int v = reinterpret_cast<const int16_t*>(S.coef[b])[zz];
              h &= h - 1;
              if (pg_bits(S, at, 1) && !(v & p1)) blk[zz] = (int16_t)(v + (v >= 0 ? p1 : m1));
            }
            if (k4 < PG_ZEND && (e & 0x10000u)) blk[S.zz[s.ss + k]] = (int16_t)(e & 0x20000u ? m1 : p1);
          }
        }
      }
      __syncthreads();
    }
    if (tid == 0) {
      // the interval ends at its first error; a value out of range precedes the symbol that ends the walk
      if (S.range < INT_MAX) S.err = CJ_DEV_DC_RANGE;
      if (S.err) cj_raise(st, pg_block(s, S, u0, bps, blk0 + min(S.done, S.range)), S.err);
      S.blk = blk0 + S.done;
      if (progress) pg_publish(progress, nscans, wk.scan, S.done);
      S.rawpos = raw0 + min((int)S.raw[min(S.pos >> 3, PG_BYTES)], (int)min((int64_t)65535, wk.end - raw0));
      S.bit = S.pos & 7;
    }
    __syncthreads();
  }
  if (progress && tid == 0) pg_publish(progress, nscans, wk.scan, nseq - S.blk);  // an error's blocks: none waits for them
}

// ---- short intervals: a thread each.  A CTA of k_prog_scans takes 8 us for an
// interval however short, and one at a time fits an SM; thousands of intervals of a
// few bytes are done sooner by a thread each, decoding symbol by symbol from global
// memory (pg_thin).

// MSB-first bits of one interval's stuffed bytes: FF 00 reads as FF; bytes
// past the end read as 0.
struct PGBits {
  const uint8_t* p;
  const uint8_t* e;
  uint64_t acc;
  int n;
  __device__ __forceinline__ void fill() {
    while (n <= 56) {
      uint32_t b = 0;
      if (p < e) {
        b = *p++;
        if (b == 0xFF && p < e && *p == 0x00) p++;
      }
      acc |= (uint64_t)b << (56 - n);
      n += 8;
    }
  }
  __device__ __forceinline__ uint32_t peek16() {
    fill();
    return (uint32_t)(acc >> 48);
  }
  __device__ __forceinline__ uint32_t bits(int k) {  // k <= 16
    if (!k) return 0;
    fill();
    const uint32_t v = (uint32_t)(acc >> (64 - k));
    acc <<= k;
    n -= k;
    return v;
  }
  // Huffman symbol, or -1 when no code matches
  __device__ __forceinline__ int huff(const CJHuff& t) {
    const uint32_t e = cj_huff_decode(t, peek16());
    if (!e) return -1;
    acc <<= (e >> 8);
    n -= (int)(e >> 8);
    return (int)(e & 255);
  }
};

// A value into an int16 coefficient; false when it does not fit.
__device__ __forceinline__ bool pg_store(int16_t* c, int v) {
  if (v < -32768 || v > 32767) return false;
  *c = (int16_t)v;
  return true;
}

// One block of a scan (T.81 G.1.2): returns 0 or a CJ_DEV_* code.
__device__ int pg_serial_block(const CJProgTables& P, int j, PGBits& br, int16_t* blk, int* dc_pred, int* eobrun,
                               const uint8_t* zz) {
  const CJProgScan& S = P.s;
  if (S.ss == 0) {
    if (!S.ah) {
      const int s = br.huff(P.huff[S.dc_slot[j]]);
      if (s < 0) return CJ_DEV_BAD_CODE;
      if (s > 11) return CJ_DEV_BAD_AC;
      dc_pred[j] += s ? cj_extend(br.bits(s), s) : 0;
      if (!pg_store(&blk[0], dc_pred[j] * (1 << S.al))) return CJ_DEV_DC_RANGE;
    } else if (br.bits(1)) {
      blk[0] = (int16_t)(blk[0] | (1 << S.al));
    }
    return 0;
  }
  const CJHuff& t = P.huff[S.ac_slot[j]];
  int k = S.ss;
  if (!S.ah) {
    if (*eobrun > 0) {
      (*eobrun)--;
      return 0;
    }
    while (k <= S.se) {
      const int rs = br.huff(t);
      if (rs < 0) return CJ_DEV_BAD_CODE;
      const int r = rs >> 4, s = rs & 15;
      if (s) {
        k += r;
        if (k > S.se) return CJ_DEV_BAD_AC;
        if (!pg_store(&blk[zz[k]], cj_extend(br.bits(s), s) * (1 << S.al))) return CJ_DEV_DC_RANGE;
        k++;
      } else if (r == 15) {
        k += 16;
      } else {
        *eobrun = (1 << r) - 1;
        if (r) *eobrun += (int)br.bits(r);
        break;
      }
    }
    return 0;
  }
  const int p1 = 1 << S.al, m1 = -(1 << S.al);
  if (*eobrun == 0) {
    for (; k <= S.se; k++) {
      const int rs = br.huff(t);
      if (rs < 0) return CJ_DEV_BAD_CODE;
      int r = rs >> 4, val = 0;
      const int s = rs & 15;
      if (s) {
        if (s != 1) return CJ_DEV_BAD_AC;
        val = br.bits(1) ? p1 : m1;
      } else if (r != 15) {
        *eobrun = 1 << r;
        if (r) *eobrun += (int)br.bits(r);
        break;
      }
      // pass r zero-history coefficients, refining the nonzero ones met
      while (k <= S.se) {
        int16_t* c = &blk[zz[k]];
        if (*c) {
          if (br.bits(1) && !(*c & p1)) *c = (int16_t)(*c + (*c >= 0 ? p1 : m1));
        } else if (--r < 0) {
          break;
        }
        k++;
      }
      if (val) {
        if (k > S.se) return CJ_DEV_BAD_AC;
        blk[zz[k]] = (int16_t)val;
      }
    }
  }
  if (*eobrun > 0) {
    // inside an end-of-band run: the correction bits of the nonzero coefficients
    for (; k <= S.se; k++) {
      int16_t* c = &blk[zz[k]];
      if (*c && br.bits(1) && !(*c & p1)) *c = (int16_t)(*c + (*c >= 0 ? p1 : m1));
    }
    (*eobrun)--;
  }
  return 0;
}

#define PG_THIN_THREADS 128
__global__ void __launch_bounds__(PG_THIN_THREADS) k_prog_thin(const CJProgTables* __restrict__ scan,
                                                              const int64_t* __restrict__ spans,
                                                              const uint8_t* __restrict__ file,
                                                              int16_t* __restrict__ coef, CJStatus* st) {
  __shared__ CJProgTables P;
  __shared__ uint8_t zz[64];
  const int iv = blockIdx.x * PG_THIN_THREADS + threadIdx.x;
#pragma unroll 10
  for (int k = threadIdx.x; k < (int)(sizeof(P) / 4); k += PG_THIN_THREADS)
    reinterpret_cast<uint32_t*>(&P)[k] = reinterpret_cast<const uint32_t*>(scan)[k];
  if (threadIdx.x < 64) zz[threadIdx.x] = c_prog_zz[threadIdx.x];
  __syncthreads();
  const CJProgScan& s = P.s;
  if (iv >= s.nint) return;
  PGBits br = {file + spans[2 * iv], file + spans[2 * iv + 1], 0, 0};
  int dc_pred[3] = {0, 0, 0}, eobrun = 0;
  const int u0 = s.ri ? iv * s.ri : 0;
  const int u1 = s.ri ? min(s.nunits, u0 + s.ri) : s.nunits;
  for (int u = u0; u < u1; u++) {
    int64_t at = (int64_t)u * s.bpm;
    if (s.ns == 1) {  // one component: its blocks in raster order
      const int bx = u % s.bw, by = u / s.bw;
      at = ((int64_t)(by / s.sy[0]) * s.mcux + bx / s.sx[0]) * s.bpm + (by % s.sy[0]) * s.sx[0] + bx % s.sx[0];
    }
    for (int j = 0; j < s.ns; j++)
      for (int w = 0; w < (s.ns > 1 ? s.sx[j] * s.sy[j] : 1); w++) {
        const int64_t blk = at + s.first[j] + w;
        const int e = pg_serial_block(P, j, br, coef + blk * 64, dc_pred, &eobrun, zz);
        if (e) {
          cj_raise(st, blk, e);
          return;
        }
      }
  }
}

// ---------------------------------------------------------------- host side

// Whether a scan's intervals are decoded by a thread each: the estimated times of both
// ways, in us.  A thread's chain is its interval's bytes and, in an AC refinement,
// the loads of every coefficient of the band in its blocks (21 us a block of the whole
// band); the CTAs run in waves of one per SM, 8.3 us each.  Fitted to 4:2:0 files of
// 128x96 to 2048x1536 samples and qualities 60 to 95; device time of all ten scans by
// CTAs / by threads at 1024x768, q 80: an interval per MCU 4.0 / 0.6 ms, per 4 MCUs
// 1.1 / 0.75, per 8 0.65 / 1.3, per 32 0.29 / 4.9; 2048x1536: per MCU 13.0 / 1.9, per
// 16 1.4 / 2.6.  `change`: what a change of way costs, where the scan before went the
// other (a launch of its own for what is noted, which then overlaps with less).
#define PG_CHANGE_US 20.0
static bool pg_thin(const CJProgScan& s, int64_t longest, int64_t bytes, int sms, double change) {
  double thread = 15.0 + 0.0066 * s.nint;
  if (!s.ah) thread += 1.5 * longest;
  else if (s.ss) thread += 4.0 * longest + 21.0 / 63 * (s.se - s.ss + 1) * (s.ri ? s.ri : s.nunits);
  else thread += 4.0 * longest;  // (eight blocks a byte)
  return thread + change < 8.0 + (8.3 * s.nint + 0.15 * bytes) / sms;
}

// Validate the SOS header of a progressive frame (T.81 B.2.3, G.1.1.1.1) at
// jpg->pos and fill `s` with the scan's components and band; on success
// jpg->pos is on the first entropy-coded byte.
int cj_parse_prog_sos(JPGReader* jpg, CJProgScan* s) {
  unsigned char* p = jpg->pos;
  if (p + 2 > jpg->end) return SYNTAX_ERROR;
  const unsigned hlen = read16(p);
  if (hlen < 6 || p + hlen > jpg->end) return SYNTAX_ERROR;
  if (!jpg->num_channels) return SYNTAX_ERROR;  // SOS before SOF
  const int ns = p[2];
  if (ns < 1 || ns > jpg->num_channels || hlen != 6u + 2u * ns) return SYNTAX_ERROR;
  memset(s, 0, sizeof(*s));
  int prev = -1;
  for (int j = 0; j < ns; j++) {
    const unsigned char* d = p + 3 + 2 * j;
    int c = 0;
    while (c < jpg->num_channels && jpg->channels[c].id != d[0]) c++;
    if (c == jpg->num_channels || c <= prev || (d[1] & 0xEE)) return SYNTAX_ERROR;
    prev = c;
    ColourChannel* ch = &jpg->channels[c];
    ch->dc_id = d[1] >> 4;
    ch->ac_id = (d[1] & 1) | 2;
    s->dc_slot[j] = ch->dc_id;
    s->ac_slot[j] = ch->ac_id;
    s->first[j] = jpg->dev->comp_first[c];
    s->sx[j] = ch->samples_x;
    s->sy[j] = ch->samples_y;
    if (ns == 1) {
      s->bw = (ch->width + 7) / 8;
      s->bh = (ch->height + 7) / 8;
    }
  }
  const unsigned char* t = p + 3 + 2 * ns;
  s->ns = ns;
  s->ss = t[0];
  s->se = t[1];
  s->ah = t[2] >> 4;
  s->al = t[2] & 15;
  if ((s->ss == 0) != (s->se == 0) || s->se > 63 || s->ss > s->se || (s->ss && ns != 1) || s->al > 13 ||
      (s->ah && s->ah != s->al + 1))
    return SYNTAX_ERROR;
  for (int j = 0; j < ns; j++) {
    const bool need_dc = s->ss == 0 && !s->ah, need_ac = s->ss != 0;
    if ((need_dc && !(jpg->huff_defined & (1 << s->dc_slot[j]))) ||
        (need_ac && !(jpg->huff_defined & (1 << s->ac_slot[j]))))
      return SYNTAX_ERROR;
  }
  jpg->pos += hlen;
  return 0;
}

static int pg_decode_noted(JPGReader* jpg);

// Queue the decode of one scan by a thread per interval.
static int pg_decode_thin(CJReaderDevice* d, const CJProgBlock& blk, const std::vector<int64_t>& spans) {
  // the block and the spans, in one stream-ordered copy: the next scan's copy into the
  // same buffer waits for this scan's kernel
  const size_t pbytes = (sizeof(CJProgTables) + 15) & ~(size_t)15, sbytes = spans.size() * sizeof(int64_t);
  std::vector<uint8_t> host(pbytes + sbytes);
  memcpy(host.data(), static_cast<const CJProgTables*>(&blk), sizeof(CJProgTables));
  memcpy(host.data() + pbytes, spans.data(), sbytes);
  if (cj_dev_ensure(d->pscan, host.size())) return CUDA_MEM_ERROR;
  CJ_CUDA_TRY(cudaMemcpyAsync(d->pscan.p, host.data(), host.size(), cudaMemcpyHostToDevice, d->stream), CUDA_MEM_ERROR);
  d->param_bytes += host.size();
  if (!d->nkev) cj_profile_begin(d);
  k_prog_thin<<<(blk.s.nint + PG_THIN_THREADS - 1) / PG_THIN_THREADS, PG_THIN_THREADS, 0, d->stream>>>(
      (const CJProgTables*)d->pscan.p, (const int64_t*)((const uint8_t*)d->pscan.p + pbytes), (const uint8_t*)d->raw.p,
      (int16_t*)d->coef.p, (CJStatus*)d->status.p);
  cj_after_launch(d, CJ_K_PROG_SCAN);
  CJ_CUDA_TRY(cudaGetLastError(), CUDA_KERNEL_LAUNCH_ERROR);
  return 0;
}

// decodeScanGPU for a scan of a progressive frame: check the header, find the
// scan's restart intervals and its end (the next marker that is not RSTn),
// and note it for the frame's pixel stage (cj_prog_finish), or for an earlier
// launch when there are many.  The first scan of the frame copies the file to the
// device and clears the coefficients.
static int pg_note_scan(JPGReader* jpg) {
  CJReaderDevice* d = jpg->dev;
  // the header first (host only, so a malformed file fails the same way
  // with or without a GPU), then the device
  for (int c = 0, k = 0; c < jpg->num_channels; c++) {
    d->comp_first[c] = k;
    k += jpg->channels[c].samples_x * jpg->channels[c].samples_y;
  }
  CJProgBlock blk;
  int err = cj_parse_prog_sos(jpg, &blk.s);
  if (err) return err;
  err = cj_gpu_init(jpg);
  if (err) return err;
  if (!d->prog_scans) cj_fill_params(jpg, (CJScanParams*)d->h_params.p);
  const CJScanParams* hp = (const CJScanParams*)d->h_params.p;
  CJProgScan& S = blk.s;
  S.bpm = hp->bpm;
  S.mcux = hp->mcux;
  S.nunits = S.ns > 1 ? hp->mcux * hp->mcuy : S.bw * S.bh;
  S.ri = jpg->restart_interval;
  S.nint = S.ri ? (S.nunits + S.ri - 1) / S.ri : 1;
  // a frame header behind the first scan does not take later ones outside the coefficient
  // buffer, which the first scan's geometry sized
  int64_t top = 0;  // the last block of the scan
  for (int j = 0; j < S.ns; j++) {
    const int64_t mcu = S.ns > 1 ? S.nunits - 1 : (int64_t)((S.bh - 1) / S.sy[0]) * S.mcux + (S.bw - 1) / S.sx[0];
    top = std::max(top, mcu * S.bpm + S.first[j] + S.sx[j] * S.sy[j] - 1);
  }
  if (top >= hp->total_blocks) return SYNTAX_ERROR;
  for (int slot = 0; slot < 4; slot++) {
    if (jpg->huff_defined & (1 << slot)) cj_build_huff(d->huff[slot].counts, d->huff[slot].symbols, &blk.huff[slot]);
    else memset(&blk.huff[slot], 0, sizeof(CJHuff));
  }
  // restart intervals and the end of the scan, from the stuffed bytes
  const unsigned char* base = jpg->buf;
  std::vector<int64_t> spans;
  // (an interval costs two bytes of file at the least, whatever the header says)
  spans.reserve(std::min(2 * (size_t)S.nint, (size_t)(jpg->end - jpg->pos) + 2));
  spans.push_back((int64_t)(jpg->pos - base));
  unsigned char* q = jpg->pos;
  const unsigned char* lim = jpg->end;  // the EOI marker lies past it
  int expect = 0;
  int64_t longest = 0;
  for (;;) {
    q = (unsigned char*)memchr(q, 0xFF, (size_t)(lim - q));
    if (!q || q + 1 >= lim + 2) {
      q = (unsigned char*)lim;
      break;
    }
    const unsigned char m = q[1];
    if (m == 0x00) {
      q += 2;
      continue;
    }
    if ((m & 0xF8) == 0xD0) {  // RSTn: ends one interval, starts the next
      if ((m & 7) != expect || (int)(spans.size() / 2) + 1 >= S.nint) return SYNTAX_ERROR;
      expect = (expect + 1) & 7;
      longest = std::max(longest, (int64_t)(q - base) - spans.back());
      spans.push_back((int64_t)(q - base));
      spans.push_back((int64_t)(q + 2 - base));
      q += 2;
      continue;
    }
    break;  // the next marker segment (or EOI)
  }
  longest = std::max(longest, (int64_t)(q - base) - spans.back());
  spans.push_back((int64_t)(q - base));
  if ((int)(spans.size() / 2) != S.nint) return SYNTAX_ERROR;
  const size_t file_bytes = (size_t)(jpg->end + 2 - base);
  if (!d->prog_scans) {
    const CJScanParams* h = hp;
    d->total_blocks = h->total_blocks;
    if (cj_dev_ensure(d->raw, file_bytes + 64) || cj_dev_ensure(d->status, sizeof(CJStatus)) ||
        cj_dev_ensure(d->coef, (size_t)d->total_blocks * 128 + 128) || cj_dev_ensure(d->params, sizeof(CJScanParams)))
      return CUDA_MEM_ERROR;
    CJ_CUDA_TRY(cudaEventRecord(d->ev_begin, d->stream), CUDA_KERNEL_LAUNCH_ERROR);
    CJ_CUDA_TRY(cudaMemcpyAsync(d->raw.p, base, file_bytes, cudaMemcpyHostToDevice, d->stream), CUDA_MEM_ERROR);
    CJ_CUDA_TRY(cudaMemsetAsync(d->coef.p, 0, (size_t)d->total_blocks * 128, d->stream), CUDA_MEM_ERROR);
    CJ_CUDA_TRY(cudaMemsetAsync(d->status.p, 0, sizeof(CJStatus), d->stream), CUDA_MEM_ERROR);
    d->raw_len = file_bytes;
    d->param_bytes = 0;
    d->nkev = 0;
  }
  if (!d->prog_scans) {  // (a file that ended in an error may have left some)
    d->prog_blocks.clear();
    d->prog_spans.clear();
    d->prog_noted = 0;
  }
  const double change = d->prog_noted ? PG_CHANGE_US : (d->prog_scans ? -PG_CHANGE_US : 0.0);
  if (pg_thin(S, longest, spans.back() - spans.front(), d->sms, change)) {  // decoded at once, behind what is noted
    err = pg_decode_noted(jpg);
    if (!err) err = pg_decode_thin(d, blk, spans);
    if (err) return err;
    d->prog_scans++;
    jpg->pos = q;
    return 0;
  }
  const uint8_t* pb = reinterpret_cast<const uint8_t*>(&blk);
  d->prog_blocks.insert(d->prog_blocks.end(), pb, pb + sizeof(blk));
  d->prog_spans.insert(d->prog_spans.end(), spans.begin(), spans.end());
  d->prog_scans++;
  d->prog_noted++;
  jpg->pos = q;  // the marker that ends the scan
  if (d->prog_noted >= PG_NOTE_SCANS || d->prog_spans.size() >= 2 * (size_t)PG_NOTE_INTERVALS) return pg_decode_noted(jpg);
  return 0;
}

// Queue the decode of the noted scans, behind that of the scans before them.
static int pg_decode_noted(JPGReader* jpg) {
  CJReaderDevice* d = jpg->dev;
  const int n = d->prog_noted;
  if (!n) return 0;
  CJProgBlock* blocks = reinterpret_cast<CJProgBlock*>(d->prog_blocks.data());
  // a scan follows the last ones before it that touch a coefficient of its; its level
  // is one more than theirs
  std::vector<int> level(n);
  int levels = 0, last[CJ_MAX_BPM][64];  // scan + 1, by the component's first block in an MCU
  bool one_launch = true;
  memset(last, 0, sizeof(last));
  for (int i = 0; i < n; i++) {
    CJProgBlock& b = blocks[i];
    const CJProgScan& s = b.s;
    b.blocks = s.nunits;
    if (s.ns > 1) {
      int bps = 0;
      for (int j = 0; j < s.ns; j++) bps += s.sx[j] * s.sy[j];
      b.blocks *= bps;
    }
    b.ndep = 0;
    b.whole = 0;
    int l = 0;
    for (int j = 0; j < s.ns; j++)
      for (int k = s.ss; k <= s.se; k++) {
        const int p = last[s.first[j]][k] - 1;
        last[s.first[j]][k] = i + 1;
        if (p < 0 || std::find(b.dep, b.dep + b.ndep, p) != b.dep + b.ndep) continue;
        if (p == i) continue;
        l = std::max(l, level[p] + 1);
        if (b.ndep == PG_DEPS) {
          one_launch = false;
          continue;
        }
        // block by block: refinements of one component's AC band, whose chunks are of PG_REF_BLOCKS
        const CJProgScan& q = blocks[p].s;
        if (!(s.ss > 0 && s.ah && q.ss > 0 && q.nint == 1 && s.nint == 1)) b.whole |= 1u << b.ndep;
        b.dep[b.ndep++] = p;
      }
    level[i] = l;
    levels = std::max(levels, l + 1);
  }
  std::vector<CJProgWork> work;
  std::vector<size_t> from(levels + 1, 0);
  for (int l = 0; l < levels; l++) {
    size_t at = 0;
    for (int i = 0; i < n; i++) {
      const CJProgScan& s = blocks[i].s;
      for (int iv = 0; iv < s.nint && level[i] == l; iv++)
        work.push_back(CJProgWork{d->prog_spans[at + 2 * iv], d->prog_spans[at + 2 * iv + 1], i, iv});
      at += 2 * (size_t)s.nint;
    }
    from[l + 1] = work.size();
  }
  CJ_CUDA_TRY(cudaFuncSetAttribute(k_prog_scans, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PGShared)),
              CUDA_KERNEL_LAUNCH_ERROR);
  int per = 0;
  CJ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_prog_scans, PG_THREADS, sizeof(PGShared)),
              CUDA_KERNEL_LAUNCH_ERROR);
  one_launch = one_launch && levels > 1 && work.size() <= (size_t)d->sms * per;
  // copied together: the scans' blocks, the work items, the progress counters' zeros
  const size_t pbytes = ((size_t)n * sizeof(CJProgBlock) + 15) & ~(size_t)15;
  const size_t wbytes = work.size() * sizeof(CJProgWork), bytes = pbytes + wbytes + (n + 1) * sizeof(int);
  d->prog_blocks.resize(bytes);
  memcpy(d->prog_blocks.data() + pbytes, work.data(), wbytes);
  memset(d->prog_blocks.data() + pbytes + wbytes, 0, (n + 1) * sizeof(int));
  if (cj_dev_ensure(d->pscan, bytes)) return CUDA_MEM_ERROR;
  CJ_CUDA_TRY(cudaMemcpyAsync(d->pscan.p, d->prog_blocks.data(), bytes, cudaMemcpyHostToDevice, d->stream),
              CUDA_MEM_ERROR);
  d->param_bytes += bytes;
  if (!d->nkev) cj_profile_begin(d);
  uint8_t* dev = (uint8_t*)d->pscan.p;
  for (int l = 0; l < (one_launch ? 1 : levels); l++) {
    const CJProgBlock* a_scans = (const CJProgBlock*)dev;
    const CJProgWork* a_work = (const CJProgWork*)(dev + pbytes) + from[l];
    const uint8_t* a_file = (const uint8_t*)d->raw.p;
    int16_t* a_coef = (int16_t*)d->coef.p;
    CJStatus* a_st = (CJStatus*)d->status.p;
    int* a_progress = one_launch ? (int*)(dev + pbytes + wbytes) : nullptr;
    int a_n = n;
    unsigned a_limit = d->wait_limit ? d->wait_limit : PG_WAIT_POLLS;
    void* args[] = {&a_scans, &a_work, &a_file, &a_coef, &a_st, &a_progress, &a_n, &a_limit};
    const unsigned grid = (unsigned)((one_launch ? work.size() : from[l + 1]) - from[l]);
    // CTAs that wait for one another are all resident (cooperative); levels need not be
    CJ_CUDA_TRY(one_launch ? cudaLaunchCooperativeKernel((const void*)k_prog_scans, dim3(grid), dim3(PG_THREADS), args,
                                                         sizeof(PGShared), d->stream)
                           : cudaLaunchKernel((const void*)k_prog_scans, dim3(grid), dim3(PG_THREADS), args,
                                              sizeof(PGShared), d->stream),
                CUDA_KERNEL_LAUNCH_ERROR);
    cj_after_launch(d, CJ_K_PROG_SCAN);
  }
  d->prog_blocks.clear();
  d->prog_spans.clear();
  d->prog_noted = 0;
  return 0;
}

// Decode the scans still noted and queue the pixel stage's parameters (geometry and
// the quantisation tables; the Huffman tables are not needed after the scans).
static int pg_finish(JPGReader* jpg) {
  CJReaderDevice* d = jpg->dev;
  const int err = pg_decode_noted(jpg);
  if (err) return err;
  CJScanParams* hp = (CJScanParams*)d->h_params.p;
  cj_fill_params(jpg, hp);
  // (the pixel stage reads as many blocks as the last frame header says)
  if (hp->total_blocks > d->total_blocks) return SYNTAX_ERROR;
  d->total_blocks = hp->total_blocks;
  CJ_CUDA_TRY(cudaMemcpyAsync(d->params.p, hp, sizeof(CJScanParams), cudaMemcpyHostToDevice, d->stream),
              CUDA_MEM_ERROR);
  CJ_CUDA_TRY(cudaEventRecord(d->ev_scan, d->stream), CUDA_KERNEL_LAUNCH_ERROR);
  return 0;
}

// (no exception leaves the library: its callers are C)
int cj_prog_scan(JPGReader* jpg) {
  try {
    return pg_note_scan(jpg);
  } catch (const std::bad_alloc&) {
    return OOM_ERROR;
  }
}

int cj_prog_finish(JPGReader* jpg) {
  try {
    return pg_finish(jpg);
  } catch (const std::bad_alloc&) {
    return OOM_ERROR;
  }
}
