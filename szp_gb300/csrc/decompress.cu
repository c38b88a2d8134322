// decompress.cu -- SZp fastmode1 / fastmode2 float32 decompressors for sm_103a.
//
// The stream keeps no block index: a block's position depends on the bit
// counts of all blocks before it in its segment (szpd_float.cc:76-118).  Three
// launches recover the positions and decode:
//
//  1. dec_setup   one CTA reads eb and the T segment offsets, validates them and
//                 cuts every segment's block region into fixed chunks.
//  2. locate      one CTA per super-chunk (threads x chunk bytes) of a segment:
//                 the bytes (plus an overlap before them) are staged in shared
//                 memory by a bulk copy and every thread walks the chain of
//                 block headers through its chunk.  Only a segment's first
//                 chunk knows where its first header is; the others start early
//                 (in the overlap) at the first position whose chain stays
//                 valid: chains started on payload bytes die within a step or
//                 two (a header byte must be <= 33) or land on a true header and
//                 follow the true chain from then on.  A chunk is right when its
//                 first header is its predecessor's exit; wrong chunks (rare)
//                 are re-walked in order.  Across CTAs a decoupled look-back
//                 sums header counts and checks the same chain property on the
//                 (entry, exit) pairs the predecessors published; a CTA whose
//                 entry proves wrong re-walks from the true one.  Each chunk then
//                 writes the header offset of each of its blocks.
//  3. decode      decode_generic: one warp per block, a look-back over the tiles
//                 of a segment for the running q (fastmode1), or each block from
//                 its seed (fastmode2).
//
// These are the passes of blockSizes other than 8, 16, ... 256, which
// decode_flow (decode_flow.cu) takes in one kernel after dec_setup.
#include <type_traits>

#include "szp_device.cuh"
#include "szp_f64.h"
#include "szp_kernels.h"
#include "szp_pipe.cuh"
#include "szp_tma.cuh"
#include "szp_unpack.cuh"

namespace szp {

constexpr uint32_t kPosEnd = 0xFFFFFFFEu;   // the walk left the segment region
constexpr uint32_t kPosDead = 0xFFFFFFFFu;  // the walk met an invalid header

// Size of a full block whose bit-count byte is b; 0 if b is not a valid
// header.  fastmode2 blocks carry a 4-byte seed and L-1 deltas.
__host__ __device__ __forceinline__ uint32_t full_block_size(uint32_t b, uint32_t L, bool fm2) {
  if (b > (uint32_t)kMaxBitCount) return 0;
  if (!fm2) return block_bytes(L, b);
  if (L == 1) return b == 0 ? 5u : 0u;
  return 4 + block_bytes(L - 1, b);
}

constexpr int kLocThreads = 128;

// A chunk may hold no header at all (a block larger than the chunk), so the
// chunk size does not depend on the block size; the overlap that lets a
// speculative walk synchronise spans at least 8 of the largest blocks.
uint32_t locate_chunk_bytes(uint32_t) { return 512; }
uint32_t locate_super_bytes(uint32_t maxsz) { return locate_chunk_bytes(maxsz) * kLocThreads; }
uint32_t locate_overlap_bytes(uint32_t maxsz) {
  uint32_t w = 2048;
  while (w < 8 * maxsz && w < 65536) w *= 2;
  return w;
}
size_t locate_smem_bytes(uint32_t super_chunk, uint32_t overlap, uint32_t maxsz) {
  return (size_t)overlap + super_chunk + maxsz + 64;
}

__device__ __forceinline__ uint64_t load_u64le(const uint8_t* p) {
  uint64_t v = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) v |= (uint64_t)p[i] << (8 * i);
  return v;
}

// ---------------------------------------------------------------------------
// 1. header -> plan
// ---------------------------------------------------------------------------
// Element e of the field's output from its code, in the launch's output kind.
__device__ void put_seed(const DecArgs& a, const DecField& fd, uint64_t e, uint32_t q, float eb, double ebd) {
  if (a.out_kind == kOutDouble) {
    reinterpret_cast<unsigned long long*>(fd.y)[e] = DequantD(ebd)(q);
  } else if (a.out_kind == kOutCodes) {
    reinterpret_cast<uint32_t*>(fd.y)[e] = q;
  } else if (a.out_kind == kOutCodesAdd) {
    int32_t* p = reinterpret_cast<int32_t*>(fd.y) + e;
    const int32_t x = *p, z = (int32_t)((uint32_t)x + q);
    *p = z;
    if (((x ^ z) & ((int32_t)q ^ z)) < 0) atomicOr(fd.err, kErrQuantRange);
  } else {
    fd.y[e] = dequant(q, eb, !isfinite(eb));
  }
}

// Shape (szp_kernels.h) of the super-chunks of a segment of nblk blocks in
// `bytes` bytes, of a launch that decodes `values` values in `total` bytes and T
// segments in all (a batch takes its fields to be like this one):
// - no more than hold 32 Ki values (empty blocks take one byte for 32 values, and
//   a CTA that meets thousands of them is the last to finish: a 2^24-value walk
//   at REL 1e-2 decodes 16 KB into 2 MB) or about 1024 blocks (the list of
//   them has 1536 places; 33.5 M values in blocks of 8 at 0.48 bytes a value: 299
//   -> 207 us);
// - where 1064 CTAs (7 on each of 152 SMs; the server runs fewer) take one or two
//   turns, as many as make these full and no third: 1 MB of floats 22 -> 18 us;
//   21.5 MB in one segment 208 -> 162 us a call (1312 super-chunks on 1064 CTAs
//   became 1955); at three turns and more smaller super-chunks lost 3 %;
// - fastmode1 blocks of 8 and 16 values: of shorter chunks, as far as that needs no more
//   than 16 of them (decode_flow.cu, kVarChunks);
// - no more chunks than leave each the room to note 5/4 of its blocks (134 M values in
//   blocks of 32 at 0.26 bytes a value: 412 -> 317 us).
__device__ __forceinline__ uint32_t flow_shape(const DecArgs& a, uint64_t bytes, uint64_t nblk, uint32_t L,
                                               uint64_t total, uint64_t values, uint64_t T) {
  // in single precision: the result only has to be the same wherever it is taken
  constexpr float kCtas = 1064.0f;
  const float blocks = (float)min(32768u >> (31 - __clz(L)), 1024u), most_values = blocks * (float)L;  // L: a power of two
  const float most = (float)(kFlowSuper / a.super_chunk), c = (float)a.super_chunk;
  const float fit = __fdiv_rn((float)bytes * blocks, fmaxf((float)nblk, 1.0f) * c);  // chunks that hold `blocks`
  const float turns = fmaxf(1.0f, ceilf(fmaxf(__fdiv_rn((float)total, kCtas * most * c),
                                              __fdiv_rn((float)values, kCtas * most_values))));
  // every segment may end in a short one
  const float slots = fmaxf(kCtas * turns - (float)T, 0.5f * kCtas * turns);
  const float by_total = turns <= 1.0f ? __fdiv_rn((float)total, 1024.0f * c)
                         : turns <= 2.0f ? ceilf(__fdiv_rn((float)total, slots * c)) : most;
  const uint32_t s = L <= 16 && !a.fm2 ? (fit <= 2.0f ? 3 : fit <= 4.0f ? 2 : fit <= 8.0f ? 1 : 0) : 0;
  const float u = (float)(1u << s);
  // whole chunks, but not above 1300 blocks
  const float by_blocks = s ? ceilf(fit * u) : fminf(ceilf(fit), floorf(fit * 1.27f));
  const float room = (float)kFlowNotes * 0.8f * fit * u;  // `blocks` times the chunks whose blocks have room
  const float by_notes = room >= 16.0f * blocks ? 16.0f : room >= 8.0f * blocks ? 8.0f : room >= 4.0f * blocks ? 4.0f
                         : room >= 2.0f * blocks ? 2.0f : 1.0f;
  const float k = fminf(fminf(by_notes, most * u), fminf(by_blocks, floorf(by_total * u)));
  return s << 4 | ((uint32_t)fmaxf(u, k) - 1);
}

template <bool BATCH>
__global__ void dec_setup_kernel(const __grid_constant__ DecArgs a) {
  const DecField& fd = BATCH ? a.fields[blockIdx.x] : a.f;
  const Segments sg = fd.seg;
  const uint32_t T = sg.T;
  const uint32_t hb = a.hb == 8 ? 8u : 4u;  // eb header: float, or double (szpd_double.cc)
  const uint64_t head = hb + 8ull * T;
  constexpr uint32_t kTurnT = 512;  // segments at most for the turns below
  __shared__ uint32_t s_cb[kTurnT + 1], s_k[kTurnT];  // tickets before each segment; its shape
  __shared__ uint32_t s_bad, s_base0, s_all, s_most;  // s_most: of the segment with the most super-chunks
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (!BATCH) {
    let_next_start();
    if (threadIdx.x == 0) {  // (a batch clears its fields' status in a launch before)
      *a.err = 0;
      a.counters[0] = 0;
    }
  }
  uint64_t len = fd.len;
  if (fd.len_dev) {
    uint64_t l2 = *fd.len_dev;
    len = l2 < len ? l2 : len;
  }
  const bool hdr_ok = len >= head;
  if (threadIdx.x == 0) s_bad = hdr_ok ? 0u : 1u;
  float eb = 0.0f;
  double ebd = 0.0;
  if (hdr_ok && (threadIdx.x == 0 || (T > sg.n && sg.tsz <= 1) || sg.tsz == 1)) {  // every thread that may write a seed
    eb = __uint_as_float((uint32_t)fd.in[0] << 24 | (uint32_t)fd.in[1] << 16 | (uint32_t)fd.in[2] << 8 | fd.in[3]);
    if (hb == 8) {
      unsigned long long d = 0;
      for (int i = 0; i < 8; i++) d = (d << 8) | fd.in[i];
      ebd = __longlong_as_double((long long)d);
    }
  }
  if (threadIdx.x == 0) {
    fd.plan->eb = eb;
    fd.plan->ebd = ebd;
  }
  // a segment's shape, in its place in a ticket
  auto shape_of = [&](uint64_t bytes, uint64_t nblk) -> uint32_t {
    return flow_shape(a, bytes, nblk, sg.L, gridDim.x * len, gridDim.x * sg.n, (uint64_t)gridDim.x * T) << kFlowPosBits;
  };
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < T; t += blockDim.x) {
    uint64_t len_t = sg.len(t);
    uint64_t r0 = 0, r1 = 0;
    uint32_t nch = 0, k = 0;
    bool bad = false;
    if (len_t > 0 && hdr_ok) {
      uint64_t off = load_u64le(fd.in + hb + 8ull * t);
      uint64_t body = len - head;
      uint64_t end;
      if (off > body) {
        bad = true;
      } else {
        uint64_t start = head + off;
        if (t + 1 < T) {
          uint64_t off2 = load_u64le(fd.in + hb + 8ull * (t + 1));
          if (off2 < off || off2 > body) bad = true;
          end = head + off2;
        } else {
          end = len;
        }
        if (!bad) {
          uint64_t nblk = a.fm2 ? (len_t + sg.L - 1) / sg.L : sg.blocks_fm1(t);
          r0 = a.fm2 ? start : start + 4;
          if (r0 > end) {
            bad = true;
          } else {
            uint64_t bound = r0 + nblk * (uint64_t)a.maxsz;
            r1 = end < bound ? end : bound;
            if (nblk > 0 && r1 <= r0) bad = true;
            if (!a.fm2 && a.map && len_t == 1) {  // a lone seed has no blocks: its value is written here
              const uint8_t* sp = fd.in + start;
              const uint32_t q = (uint32_t)sp[0] | (uint32_t)sp[1] << 8 | (uint32_t)sp[2] << 16 | (uint32_t)sp[3] << 24;
              put_seed(a, fd, sg.lo(t), q, eb, ebd);
            }
            if (r1 - r0 >= (1ull << 32)) bad = true;  // block offsets are 32-bit
            uint32_t sc = a.super_chunk;
            if (a.map) {
              k = shape_of(r1 - r0, nblk);
              const uint32_t shape = k >> kFlowPosBits;
              sc = ((shape & 15) + 1) * (sc >> (shape >> 4));
            }
            nch = (uint32_t)((r1 - r0 + sc - 1) / sc);
          }
        }
      }
    }
    if (bad) {
      atomicOr(&s_bad, 1u);
      nch = 0;
    }
    fd.reg0[t] = r0;
    fd.reg1[t] = r1;
    if (t < kTurnT) {
      s_cb[t + 1] = nch;
      s_k[t] = k;
    } else {
      fd.chunk_base[t + 1] = nch;
    }
  }
  __syncthreads();
  if (warp == 0) {  // chunk counts -> the chunks before each segment
    uint32_t acc = 0, most = 0;
    if (lane == 0) fd.chunk_base[0] = s_cb[0] = 0;
    for (uint32_t t0 = 0; t0 < T; t0 += 128) {  // four groups of loads in flight
      uint32_t n[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t t = t0 + 32 * u + lane;
        n[u] = t >= T || s_bad ? 0u : t < kTurnT ? s_cb[t + 1] : fd.chunk_base[t + 1];
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t t = t0 + 32 * u + lane;
        if (t0 + 32 * u >= T) break;
        const uint32_t incl = acc + warp_incl_scan(n[u], lane);
        most = max(most, __reduce_max_sync(0xffffffffu, n[u]));
        if (t < T) fd.chunk_base[t + 1] = incl;
        if (t < T && t < kTurnT) s_cb[t + 1] = incl;
        acc = __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    if (lane == 0) {
      if (s_bad) atomicOr(fd.err, kErrCorrupt);
      fd.plan->nchunks = acc;
      fd.plan->bad = s_bad;
      s_all = acc;
      s_most = most;
      s_base0 = BATCH ? atomicAdd(a.ticket_total, acc) : 0u;  // the field's first ticket
    }
  }
  if (!a.map) return;
  __syncthreads();
  const uint32_t all = s_all;
  if (all == 0) return;
  // The tickets of decode_flow: field, segment, position in it, look-back
  // record (the records of a segment follow one another).  The segments take
  // turns (first super-chunk of each, second of each, ...), so that the CTAs in
  // flight stand near the fronts of all of them and a look-back has 1/T of
  // them before it (a 512^3 field at T = 16: 0.373 -> 0.291 ms); what a segment
  // has beyond 5/4 of the average comes last.
  const uint32_t turns = T < 4 || T > kTurnT ? 0u : min(all, (all + all / 4 + T - 1) / T);
  for (uint32_t j = warp; j < turns; j += nwarps) {
    uint32_t at = s_base0;  // and the tickets of the turns before j
    for (uint32_t t = lane; t < ((T + 31) & ~31u); t += 32)
      at += __reduce_add_sync(0xffffffffu, t < T ? min(s_cb[t + 1] - s_cb[t], j) : 0u);
    for (uint32_t t = lane; t < ((T + 31) & ~31u); t += 32) {
      const uint32_t c0 = s_cb[min(t, T)], n = t < T ? s_cb[t + 1] - c0 : 0u;
      const uint32_t has = __ballot_sync(0xffffffffu, n > j);
      if (n > j)
        a.map[at + __popc(has & ((1u << lane) - 1u))] = make_uint4(blockIdx.x, t, s_k[t] | j, s_base0 + c0 + j);
      at += __popc(has);
    }
  }
  if (turns == 0) {  // segment by segment: the CTA each, or a thread each where there are many
    const bool wide = T < 4;
    for (uint32_t t = wide ? 0 : threadIdx.x; t < T; t += wide ? 1 : blockDim.x) {
      const uint32_t c0 = t < kTurnT ? s_cb[t] : fd.chunk_base[t];
      const uint32_t n = (t < kTurnT ? s_cb[t + 1] : fd.chunk_base[t + 1]) - c0;
      if (n == 0) continue;
      const uint64_t len_t = sg.len(t);
      const uint32_t k = t < kTurnT ? s_k[t]
                                    : shape_of(fd.reg1[t] - fd.reg0[t], a.fm2 ? (len_t + sg.L - 1) / sg.L : sg.blocks_fm1(t));
      for (uint32_t j = wide ? threadIdx.x : 0; j < n; j += wide ? blockDim.x : 1)
        a.map[s_base0 + c0 + j] = make_uint4(blockIdx.x, t, k | j, s_base0 + c0 + j);
    }
    return;
  }
  // the rest, segment by segment; they come after the tickets of the turns
  if (s_most <= turns) return;
  uint32_t at = s_base0;
  for (uint32_t t = 0; t < T; t++) at += min(s_cb[t + 1] - s_cb[t], turns);
  for (uint32_t t = 0; t < T; t++) {
    const uint32_t c0 = s_cb[t], n = s_cb[t + 1] - c0;
    for (uint32_t j = turns + threadIdx.x; j < n; j += blockDim.x)
      a.map[at + (j - turns)] = make_uint4(blockIdx.x, t, s_k[t] | j, s_base0 + c0 + j);
    at += n > turns ? n - turns : 0u;
  }
}

// Global block index of block 0 of segment t (segments 0..T-2 are alike).
__device__ __forceinline__ uint64_t seg_block_base(const Segments& sg, uint32_t t, bool fm2) {
  uint64_t per = fm2 ? (sg.tsz + sg.L - 1) / sg.L : (sg.tsz > 1 ? (sg.tsz - 1 + sg.L - 1) / sg.L : 0);
  return (uint64_t)t * per;
}
__device__ __forceinline__ uint64_t seg_blocks(const Segments& sg, uint32_t t, bool fm2) {
  return fm2 ? (sg.len(t) + sg.L - 1) / sg.L : sg.blocks_fm1(t);
}

// ---------------------------------------------------------------------------
// 2. locate block headers
// ---------------------------------------------------------------------------
constexpr uint64_t kFlagRepair = 3;  // status: the CTA is re-walking; not ready

// CTA (super-chunk) of ticket c: largest t with chunk_base[t] <= c.
__device__ __forceinline__ uint32_t chunk_segment(const uint32_t* __restrict__ cb, uint32_t T, uint32_t c) {
  uint32_t lo_t = 0, hi_t = T - 1;
  while (lo_t < hi_t) {
    uint32_t mid = (lo_t + hi_t + 1) >> 1;
    if (cb[mid] <= c) lo_t = mid; else hi_t = mid - 1;
  }
  return lo_t;
}

// A header chain walked in the shared-memory copy of a segment's region:
// region offset p is at sb[p - base0]; bytes exist below `avail`.
struct SmemChain {
  const uint8_t* sb;
  uint32_t base0, avail, rlen, L;
  uint32_t l8;  // L / 8 for fastmode1 with L % 8 == 0 (block size 1 + l8*(b+1)), else 0
  bool fm2;
  // block size at p, 0 when its bit-count byte is invalid or not staged
  __device__ __forceinline__ uint32_t step(uint32_t p) const {
    const uint32_t skip = fm2 ? 4u : 0u;
    if (p >= avail || avail - p <= skip) return 0;
    const uint32_t b = sb[p + skip - base0];
    if (l8) return b > (uint32_t)kMaxBitCount ? 0u : (b ? 1 + l8 * (b + 1) : 1u);
    return full_block_size(b, L, fm2);
  }
  // the position sz bytes on; past 2^32 (a region may end a byte below it) the last one there is
  static __device__ __forceinline__ uint32_t after(uint32_t p, uint32_t sz) { return p + min(sz, 0xFFFFFFFFu - p); }
  // walk from p to cE: header count, exit (kPosEnd past the region, kPosDead)
  __device__ __forceinline__ uint32_t walk(uint32_t p, uint32_t cE, uint32_t* exit) const {
    uint32_t k = 0;
    while (p < cE) {
      uint32_t sz = step(p);
      if (!sz) {
        *exit = kPosDead;
        return k;
      }
      k++;
      p = after(p, sz);
    }
    *exit = p >= rlen ? kPosEnd : p;
    return k;
  }
};


// Re-walks, in order, every chunk from `from` on whose first header is not
// the exit of the chunk before it (e = exit before chunk `from`); thread-serial.
__device__ __forceinline__ void rewalk_from(const SmemChain& ch, uint32_t* h, uint32_t* x, uint32_t* k,
                                            uint32_t from, uint32_t e, uint32_t nactive, uint32_t scS,
                                            uint32_t scE, uint32_t C) {
  for (uint32_t i = from; i < nactive; i++) {
    if (e == kPosEnd || e == kPosDead) {
      h[i] = e;
      x[i] = e;
      k[i] = 0;
      continue;
    }
    if (h[i] != e) {
      const uint32_t cE = scS + min((i + 1) * C, scE - scS);
      h[i] = e;
      uint32_t ex;
      k[i] = ch.walk(e, cE, &ex);
      x[i] = ex;
    }
    e = x[i];
  }
}

// PACK: a super-chunk's look-back word carries its (entry, exit) pair too, so
// one load reads a predecessor (blocks of at most 254 bytes, super-chunks
// below 2^17 - 2 bytes).  An aggregate's 42-bit value holds the header count
// (17 bits), the entry relative to the super-chunk's start (17 bits) and the
// exit relative to its end (8 bits); an inclusive value holds the count
// prefix and the exit.  Otherwise the pair sits in a second word, read between
// two reads of the status word.
constexpr uint32_t kRelDead = 0x1FFFFu, kRelEnd = 0x1FFFEu, kXDead = 0xFFu, kXEnd = 0xFEu;

__device__ __forceinline__ uint64_t loc_word(uint64_t cnt, uint32_t h0, uint32_t xl, uint32_t scS, uint32_t scE,
                                             bool incl) {
  const uint64_t xr = xl == kPosDead ? kXDead : xl == kPosEnd ? kXEnd : (uint64_t)(xl - scE);
  if (incl) return (cnt << 8) | xr;
  const uint64_t hr = h0 == kPosDead ? kRelDead : h0 == kPosEnd ? kRelEnd : (uint64_t)(h0 - scS);
  return (cnt << 25) | (hr << 8) | xr;
}

static bool locate_packs(uint32_t super_chunk, uint32_t maxsz) {
  return maxsz <= 254 && (uint64_t)super_chunk + maxsz < kRelEnd;
}

template <bool FM2, bool PACK>
__global__ void __launch_bounds__(kLocThreads) locate_kernel(const __grid_constant__ DecArgs a) {
  constexpr int NT = kLocThreads;
  extern __shared__ __align__(16) uint8_t s_bytes[];
  __shared__ uint32_t s_tk[2];
  __shared__ uint32_t s_h[NT], s_x[NT], s_k[NT];
  __shared__ uint64_t s_val[1];
  __shared__ uint32_t s_misc[2 * (NT / 32)];
  __shared__ __align__(8) uint64_t s_bar;
  uint32_t tile, epoch;
  draw_ticket(a.ls, a.nlocate_ctas, tile, epoch, s_tk);
  const DecField& fd = a.f;
  const uint32_t lt = tile;
  const uint32_t nct = fd.plan->bad ? 0 : fd.chunk_base[fd.seg.T];
  if (lt >= nct) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Segments sg = fd.seg;
  const uint32_t t = chunk_segment(fd.chunk_base, sg.T, lt);
  const uint32_t first = fd.chunk_base[t];  // ticket of the segment's first chunk
  const uint32_t j = tile - first;
  const uint64_t R0 = fd.reg0[t];
  const uint32_t rlen = (uint32_t)(fd.reg1[t] - R0);
  const uint32_t C = a.chunk, SC = a.super_chunk, W0 = a.overlap;
  const uint32_t scS = j * SC, scE = scS + min(SC, rlen - scS);

  // ---- stage [scS - W0, scE + maxsz) of the region ----
  const uint32_t st0 = scS > W0 ? scS - W0 : 0u;
  const uint32_t st1 = (uint32_t)min((uint64_t)rlen, (uint64_t)scE + a.maxsz + 8);
  const uint8_t* g = fd.in + R0 + st0;
  const uint32_t align = (uint32_t)((uintptr_t)g & 15);
  {
    if (tid == 0) mbar_init(&s_bar, 1);
    __syncthreads();
    const uint32_t end = align + (st1 - st0);
    const uint32_t i0 = (align + 15) & ~15u, i1 = end & ~15u;
    const uint8_t* g0 = g - align;
    const bool bulk = i1 > i0;
    if (tid == 0 && bulk) {
      mbar_arrive_expect_tx(&s_bar, i1 - i0);
      bulk_load(s_bytes + i0, g0 + i0, i1 - i0, &s_bar);
    }
    if (bulk) {
      for (uint32_t b = align + tid; b < i0; b += NT) s_bytes[b] = __ldg(g0 + b);
      for (uint32_t b = i1 + tid; b < end; b += NT) s_bytes[b] = __ldg(g0 + b);
    } else {
      for (uint32_t b = align + tid; b < end; b += NT) s_bytes[b] = __ldg(g0 + b);
    }
    if (bulk && !mbar_wait_ns(&s_bar, 0, kWaitNs)) {
      atomicOr(a.err, kErrLookbackTimeout);
      mbar_wait_ns(&s_bar, 0, kWaitNs);  // the copy lands before the CTA may exit
    }
    __syncthreads();
  }
  SmemChain ch;
  ch.sb = s_bytes + align;
  ch.base0 = st0;
  ch.avail = st1;
  ch.rlen = rlen;
  ch.L = sg.L;
  ch.l8 = (!FM2 && sg.L % 8 == 0) ? sg.L / 8 : 0u;
  ch.fm2 = FM2;

  // ---- speculative walk of each thread's chunk ----
  // A lane's chain starts at `anchor` (a segment's first chunk: at its first
  // header); the first position >= cS on it is the chunk's entry, headers in
  // [cS, cE) are counted, and the first position >= cE is its exit.  A chain
  // that meets an invalid header restarts one byte after its anchor.  Each
  // lane runs its own loop of single header steps: lanes finish at different
  // times, but an iteration is a handful of instructions (a lockstep loop that
  // applied every outcome with selects cost several times as much).
  const uint32_t nactive = (scE - scS + C - 1) / C;
  const uint32_t cS = scS + tid * C, cE = (uint32_t)tid < nactive ? cS + min(C, scE - cS) : scE;
  uint32_t h = kPosEnd, x = kPosEnd, k = 0;
  if ((uint32_t)tid < nactive) {
    const bool known = j == 0 && tid == 0;  // a segment's block region starts with a header
    // a wrong guess is caught by the chain checks (inside the CTA, or across
    // CTAs for its first chunk) and re-walked from the true exit
    const uint32_t W = min(W0, max(512u, 4 * a.maxsz));
    uint32_t anchor = known ? 0u : (cS > st0 + W ? cS - W : st0);
    uint32_t pos = anchor, entry = anchor >= cS ? anchor : kPosDead, cnt = 0;
    uint32_t budget = 4 * (W + C);
    bool broken = false;
    h = kPosDead;
    x = kPosDead;
    const uint8_t* sb = ch.sb - ch.base0;  // region offset p at sb[p]
    const bool b32 = !FM2 && ch.l8 == 4;  // blockSize 32: a block of 1 or 4b + 5 bytes
    while (pos < cE && budget != 0) {
      budget--;
      // every position read is below cE, inside the staged bytes
      const uint32_t b = sb[pos];
      const uint32_t sz = b32 ? (b > (uint32_t)kMaxBitCount ? 0u : (b ? 4 * b + 5 : 1u)) : ch.step(pos);
      if (sz) {
        cnt += pos >= cS ? 1u : 0u;
        const uint32_t np = SmemChain::after(pos, sz);
        if (entry == kPosDead && np >= cS) entry = np;
        pos = np;
      } else if (!known && anchor + 1 < cE) {
        anchor++;
        pos = anchor;
        cnt = 0;
        entry = anchor >= cS ? anchor : kPosDead;
      } else {
        broken = true;
        break;
      }
    }
    if (pos >= cE) {
      h = entry >= rlen ? kPosEnd : entry;
      x = pos >= rlen ? kPosEnd : pos;
      k = cnt;
    } else if (broken && known) {
      h = 0;
      k = cnt;  // x stays kPosDead: the true chain is broken
    }
  }
  s_h[tid] = h;
  s_x[tid] = x;
  s_k[tid] = k;
  __syncthreads();
  // ---- chunk boundaries inside the CTA ----
  bool bad = false;
  if (tid > 0 && (uint32_t)tid < nactive) {
    const uint32_t px = s_x[tid - 1];
    bad = (px == kPosEnd) ? (h != kPosEnd || k != 0) : (px != h);
  }
  const uint32_t repairs = __syncthreads_count(bad);
  if (repairs) {
    if (tid == 0) {
      rewalk_from(ch, s_h, s_x, s_k, 1, s_x[0], nactive, scS, scE, C);
      atomicAdd(&a.counters[0], repairs);
    }
    __syncthreads();
  }

  // ---- look-back over header counts, verifying entries (warp 0; the
  // other warps wait at the barrier after it) ----
  uint32_t K = 0;
  for (int i = 0; i < NT; i++) K += s_k[i];  // shared reads, same in every thread
  uint32_t h0 = s_h[0], xl = s_x[nactive - 1];
  uint64_t prefix = 0;
  if (j == 0) {
    if (tid == 0) {
      if (PACK) {
        st_relaxed_u64(a.status + tile, make_status(epoch, kFlagInclusive, loc_word(K, h0, xl, scS, scE, true)));
      } else {
        a.aux[tile] = make_uint2(h0, xl);
        __threadfence();
        st_release_u64(a.status + tile, make_status(epoch, kFlagInclusive, K));
      }
    }
  } else {
    if (tid == 0) {
      if (PACK) {
        st_relaxed_u64(a.status + tile, make_status(epoch, kFlagAggregate, loc_word(K, h0, xl, scS, scE, false)));
      } else {
        a.aux[tile] = make_uint2(h0, xl);
        __threadfence();
        st_release_u64(a.status + tile, make_status(epoch, kFlagAggregate, K));
      }
    }
    if (warp == 0) {
      // lane l reads tile base - l (seqlock read of status + aux); a window
      // whose entries are not all ready, or whose chain of (entry, exit)
      // pairs is broken (an older tile will repair itself), is read again
      // after a pause
      uint32_t spins = 0;
      int verdict = 0;  // 1 done, 2 retry, 3 repair self
      uint64_t acc = 0;
      uint32_t pred_x = kPosDead;
      while (true) {
        int64_t base = (int64_t)tile - 1;
        uint32_t need_x = h0;  // exit the next-older tile must have
        bool self_ok = true;
        acc = 0;
        while (true) {
          const int64_t idx = base - lane;
          const bool inr = idx >= (int64_t)first;
          uint64_t s1 = 0, cnt = 0;
          uint2 ax = make_uint2(0, 0);
          bool ready = true, incl = false;
          if (inr) {
            if (PACK) {
              s1 = ld_volatile_u64(a.status + idx);
              const uint64_t f = status_flag(s1);
              ready = status_epoch(s1) == (epoch & 0xFFFFF) && (f == kFlagAggregate || f == kFlagInclusive);
              incl = ready && f == kFlagInclusive;
              const uint64_t v = status_value(s1);
              const uint32_t sS = (uint32_t)(idx - (int64_t)first) * SC, sE = sS + min(SC, rlen - sS);
              const uint32_t xr = (uint32_t)v & 0xFFu;
              ax.y = xr == kXDead ? kPosDead : xr == kXEnd ? kPosEnd : sE + xr;
              if (incl) {
                cnt = v >> 8;
              } else {
                const uint32_t hr = (uint32_t)(v >> 8) & 0x1FFFFu;
                ax.x = hr == kRelDead ? kPosDead : hr == kRelEnd ? kPosEnd : sS + hr;
                cnt = v >> 25;
              }
            } else {
              // acquire loads keep the aux read between the two status reads
              s1 = ld_acquire_u64(a.status + idx);
              const uint64_t axw = ld_acquire_u64(reinterpret_cast<const uint64_t*>(a.aux + idx));
              ax = make_uint2((uint32_t)axw, (uint32_t)(axw >> 32));
              const uint64_t s2 = ld_volatile_u64(a.status + idx);
              const uint64_t f = status_flag(s1);
              ready = s1 == s2 && status_epoch(s1) == (epoch & 0xFFFFF) && (f == kFlagAggregate || f == kFlagInclusive);
              incl = ready && f == kFlagInclusive;
              cnt = status_value(s1);
            }
          }
          const uint32_t bi = __ballot_sync(0xffffffffu, incl);
          const int jstar = bi ? __ffs(bi) - 1 : 32;  // nearest inclusive of the window
          const bool relevant = inr && lane <= jstar;
          if (__any_sync(0xffffffffu, relevant && !ready)) {
            verdict = 2;
            break;
          }
          // the entry of lane l's tile must be the exit of the next older
          // tile (lane l + 1); the inclusive tile is already verified
          const uint32_t ox = __shfl_down_sync(0xffffffffu, ax.y, 1);
          bool bad = false;
          if (relevant && lane < jstar && lane < 31 && idx - 1 >= (int64_t)first)
            bad = (ox == kPosEnd) ? (ax.x != kPosEnd) : (ax.x != ox);
          if (__any_sync(0xffffffffu, bad)) {
            verdict = 2;
            break;
          }
          const uint32_t px = __shfl_sync(0xffffffffu, ax.y, 0);
          if (base == (int64_t)tile - 1) {
            // our own entry against the nearest predecessor's exit
            self_ok = (px == kPosEnd) ? (h0 == kPosEnd && K == 0) : (px == h0);
            pred_x = px;
          } else if (!((px == kPosEnd) ? (need_x == kPosEnd) : (px == need_x))) {
            // window boundary: the nearest of this window must exit where the
            // farthest of the previous window entered
            verdict = 2;
            break;
          }
          uint64_t v = relevant ? cnt : 0;
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          acc += v;
          const uint32_t far_h = __shfl_sync(0xffffffffu, ax.x, 31);
          if (jstar < 32 || base - 32 < (int64_t)first) {
            verdict = self_ok ? 1 : 3;
            break;
          }
          need_x = far_h;
          base -= 32;
        }
        if (verdict != 2) break;
        if (++spins > kSpinLimit) {
          if (lane == 0) atomicOr(a.err, kErrLookbackTimeout);
          break;
        }
        __nanosleep(200);
      }
      if (lane == 0) {
        s_misc[0] = (uint32_t)verdict;
        s_misc[1] = pred_x;
        s_val[0] = acc;
      }
    }
    __syncthreads();
    const int verdict = (int)s_misc[0];
    const uint32_t pred_x = s_misc[1];
    const uint64_t acc = s_val[0];
    __syncthreads();  // s_misc and s_val are reused below
    if (verdict == 3) {
      // our speculative entry was wrong: re-walk from the verified exit
      if (tid == 0) {
        if (PACK) {
          st_relaxed_u64(a.status + tile, make_status(epoch, kFlagRepair, 0));
        } else {
          st_release_u64(a.status + tile, make_status(epoch, kFlagRepair, 0));
          __threadfence();
        }
        s_h[0] = pred_x == kPosDead ? kPosEnd : kPosDead;  // differs from the entry: chunk 0 is re-walked
        rewalk_from(ch, s_h, s_x, s_k, 0, pred_x, nactive, scS, scE, C);
        atomicAdd(&a.counters[0], 1u);
      }
      __syncthreads();
      K = 0;
      for (int i = 0; i < NT; i++) K += s_k[i];
      h0 = s_h[0];
      xl = s_x[nactive - 1];
      if (tid == 0 && !PACK) {
        a.aux[tile] = make_uint2(h0, xl);
        __threadfence();
      }
    }
    prefix = acc;
    if (tid == 0) {
      if (PACK) {
        st_relaxed_u64(a.status + tile, make_status(epoch, kFlagInclusive, loc_word(prefix + K, h0, xl, scS, scE, true)));
      } else {
        st_release_u64(a.status + tile, make_status(epoch, kFlagInclusive, prefix + K));
      }
    }
  }
  // ---- header offsets of every block of every chunk ----
  uint32_t kx = s_k[tid];
  uint32_t incl_k = kx;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, incl_k, o);
    if (lane >= o) incl_k += y;
  }
  if (lane == 31) s_misc[warp] = incl_k;
  __syncthreads();
  uint32_t wex = 0;
  for (int w = 0; w < warp; w++) wex += s_misc[w];
  const uint64_t g0 = prefix + wex + (incl_k - kx);
  const uint64_t gb = seg_block_base(sg, t, FM2), nb = seg_blocks(sg, t, FM2);
  uint32_t p = s_h[tid];
  if (kx && p < rlen) {
    for (uint32_t i = 0; i < kx; i++) {
      const uint64_t gi = g0 + i;
      if (gi < nb) fd.blkpos[gb + gi] = p;
      const uint32_t sz = ch.step(p);
      if (!sz) break;
      p += sz;
    }
  }
  // the last CTA of a segment checks the block total
  if (tid == 0 && lt + 1 == fd.chunk_base[t + 1]) {
    const uint64_t total = prefix + K;
    const bool last_seg = t + 1 == sg.T;
    if (total < nb || (!last_seg && total != nb)) atomicOr(fd.err, kErrBlockCount);
  }
}

// ---------------------------------------------------------------------------
// 3. decode
// ---------------------------------------------------------------------------

// Delta of element j of a block whose bit-count byte is at hdr (m elements).
__device__ __forceinline__ uint32_t decode_delta(const uint8_t* __restrict__ hdr, uint32_t m, uint32_t bc,
                                                 uint32_t j) {
  const uint32_t ns = (m + 7) >> 3, B = bc >> 3, r = bc & 7;
  uint32_t neg = (__ldg(hdr + 1 + (j >> 3)) >> (7 - (j & 7))) & 1u;
  const uint8_t* bp = hdr + 1 + ns;
  uint32_t hi = 0;
  if (B) {
    const uint8_t* q = bp + j * B;
    hi = __ldg(q);
    if (B > 1) hi |= (uint32_t)__ldg(q + 1) << 8;
    if (B > 2) hi |= (uint32_t)__ldg(q + 2) << 16;
    if (B > 3) hi |= (uint32_t)__ldg(q + 3) << 24;
  }
  uint32_t lo = 0;
  if (r) {
    const uint8_t* rp = bp + B * m;
    uint32_t bit = j * r;
    uint32_t off = bit & 7;
    uint32_t w = (uint32_t)__ldg(rp + (bit >> 3)) << 8;
    if (off + r > 8) w |= __ldg(rp + (bit >> 3) + 1);
    lo = (w >> (16 - off - r)) & ((1u << r) - 1u);
  }
  uint32_t v = (B ? (hi << r) : 0u) | lo;
  return neg ? 0u - v : v;
}

template <int WARPS>
__device__ __forceinline__ uint32_t scan_warps_u32(uint32_t* s_w, uint32_t mine, int warp, int lane,
                                                   uint32_t& excl) {
  if (lane == 0) s_w[warp] = mine;
  __syncthreads();
  if (warp == 0) {
    uint32_t x = lane < WARPS ? s_w[lane] : 0;
    uint32_t incl = warp_incl_scan(x, lane);
    if (lane < WARPS) s_w[lane] = incl - x;
    if (lane == 31) s_w[WARPS] = incl;
  }
  __syncthreads();
  excl = s_w[warp];
  return s_w[WARPS];
}

struct DecTile {
  uint32_t seg;
  uint64_t blk0;
  uint32_t nblk;
  bool first;
  bool any;
};

__device__ __forceinline__ DecTile dec_tile(const Segments& sg, uint32_t tile, uint32_t tiles_per_seg, uint32_t tb,
                                           bool fm2) {
  DecTile d;
  uint32_t t, ts;
  if (tiles_per_seg) {
    t = tile / tiles_per_seg;
    if (t > sg.T - 1) t = sg.T - 1;
    ts = tile - t * tiles_per_seg;
  } else {
    t = sg.T - 1;
    ts = tile;
  }
  uint64_t nb = seg_blocks(sg, t, fm2);
  d.seg = t;
  d.blk0 = (uint64_t)ts * tb;
  uint64_t rem = nb > d.blk0 ? nb - d.blk0 : 0;
  d.nblk = (uint32_t)(rem < tb ? rem : tb);
  d.first = ts == 0;
  d.any = sg.n > 0 && sg.len(t) > 0;
  return d;
}


constexpr int kDecWarps = 8;
// Any blockSize, fastmode1 or fastmode2: one warp per block in 32-element
// pieces.  fastmode1 decodes twice (totals, then values after the look-back).
// V = float, or double for float64 streams (x' = (double)q * eb).
template <int WARPS, bool FM2, typename V = float>
__global__ void __launch_bounds__(WARPS * 32) decode_generic(const __grid_constant__ DecArgs a) {
  constexpr bool DBL = std::is_same<V, double>::value;
  const DecField& fd = a.f;
  __shared__ uint32_t s_tk[2];
  __shared__ uint32_t s_w[WARPS + 1];
  __shared__ uint32_t s_base;
  uint32_t tile, epoch;
  draw_ticket(a.ls, a.ntiles, tile, epoch, s_tk);
  if (fd.plan->bad) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Segments sg = fd.seg;
  const uint32_t L = sg.L;
  const uint32_t TB = WARPS * a.bpw;
  const DecTile dt = dec_tile(sg, tile, fd.tiles_per_seg, TB, FM2);
  if (!dt.any) return;
  V eb;
  if constexpr (DBL) eb = fd.plan->ebd;
  else eb = fd.plan->eb;
  const bool ebsp = !isfinite(eb);
  // float64: (double)q * eb in integer arithmetic for every eb whose
  // products stay normal (FP64 instructions are slow on this GPU)
  bool fastdq = false;
  uint64_t ebm = 0, ebs = 0;
  uint32_t ebe = 0;
  if constexpr (DBL) {
    const uint64_t u = f64i::bits_of(eb);
    fastdq = f64i::dequant_fast_ok(u);
    ebm = (u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    ebe = (uint32_t)(u >> 52) & 0x7FFu;
    ebs = u & 0x8000000000000000ull;
  }
  auto dq = [&](uint32_t q) -> V {
    if constexpr (DBL) {
      if (fastdq) return f64i::double_of(f64i::dequant_bits((int32_t)q, ebm, ebe, ebs));
    }
    return dequant(q, eb, ebsp);
  };
  V* __restrict__ yv = DBL ? reinterpret_cast<V*>(fd.yd) : reinterpret_cast<V*>(fd.y);
  const uint64_t lo = sg.lo(dt.seg), hi = sg.hi(dt.seg);
  const uint64_t R0 = fd.reg0[dt.seg], R1 = fd.reg1[dt.seg];
  const uint8_t* __restrict__ in = fd.in;
  const uint64_t gb = seg_block_base(sg, dt.seg, FM2);
  const uint32_t wfirst = warp * a.bpw;
  bool corrupt = false;

  // elements of block b: fastmode1 [lo+1+bL, +L), fastmode2 seed at lo+bL then L-1
  auto blk_start = [&](uint64_t b) -> uint64_t { return FM2 ? lo + b * L + 1 : lo + 1 + b * L; };
  auto blk_len = [&](uint64_t b) -> uint32_t {
    uint64_t s = blk_start(b);
    uint64_t e = s + (FM2 ? L - 1 : L);
    if (e > hi) e = hi;
    return e > s ? (uint32_t)(e - s) : 0u;
  };
  // block header pointer and validation; returns bc or 255 when corrupt
  auto blk_hdr = [&](uint64_t b, uint32_t m, uint64_t& hp) -> uint32_t {
    hp = R0 + __ldg(fd.blkpos + gb + b) + (FM2 ? 4 : 0);
    if (FM2 && m == 0) return 0;  // one-element block: no header is read (szpd_float.cc:483)
    if (hp >= R1) return 255u;
    uint32_t bc = __ldg(in + hp);
    if (bc > 33 || hp + block_bytes(m, bc) > R1) return 255u;
    return bc;
  };

  // fastmode1 decodes every delta twice (the warp's total, then the values
  // once its base is known); with blockSize <= 32 (one piece per block) and
  // at most KC blocks per warp, lane c fetches block c's position and header
  // byte, the deltas of all the warp's blocks are decoded with their loads
  // in flight together, and each lane keeps its deltas in registers
  constexpr int KC = 8;
  const bool cache = !FM2 && L <= 32 && a.bpw <= (uint32_t)KC;
  uint32_t cd[KC];
#pragma unroll
  for (int c = 0; c < KC; c++) cd[c] = 0;
  uint32_t q0 = 0;
  if (!FM2) {
    uint32_t wtot = 0;
    if (cache) {
      uint64_t hpl = 0;
      uint32_t bcl = 0, ml = 0;
      if ((uint32_t)lane < a.bpw && wfirst + lane < dt.nblk) {
        ml = blk_len(dt.blk0 + wfirst + lane);
        bcl = blk_hdr(dt.blk0 + wfirst + lane, ml, hpl);
        if (bcl == 255u) {
          corrupt = true;
          bcl = 0;
        }
      }
      uint32_t lsum = 0;
#pragma unroll
      for (int c = 0; c < KC; c++) {
        if ((uint32_t)c >= a.bpw || wfirst + c >= dt.nblk) break;
        const uint32_t bc = __shfl_sync(0xffffffffu, bcl, c), m = __shfl_sync(0xffffffffu, ml, c);
        const uint64_t hp = __shfl_sync(0xffffffffu, (unsigned long long)hpl, c);
        cd[c] = (bc && (uint32_t)lane < m) ? decode_delta(in + hp, m, bc, lane) : 0u;
        lsum += cd[c];
      }
      for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
      wtot = lsum;
    }
    for (uint32_t k = 0; !cache && k < a.bpw; k++) {
      uint32_t bi = wfirst + k;
      if (bi >= dt.nblk) break;
      uint64_t b = dt.blk0 + bi, hp;
      uint32_t m = blk_len(b);
      uint32_t bc = blk_hdr(b, m, hp);
      if (bc == 255u) {
        corrupt = true;
        continue;
      }
      if (!bc) continue;
      for (uint32_t p0 = 0; p0 < m; p0 += 32) {
        uint32_t j = p0 + lane;
        uint32_t d = j < m ? decode_delta(in + hp, m, bc, j) : 0u;
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        wtot += d;
      }
    }
    uint32_t wexcl;
    const uint32_t agg = scan_warps_u32<WARPS>(s_w, wtot, warp, lane, wexcl);
    const uint32_t first_tile = fd.tiles_per_seg ? dt.seg * fd.tiles_per_seg : 0;
    if (warp == 0) {
      uint32_t excl;
      if (dt.first) {
        const uint8_t* sp = in + R0 - 4;
        excl = (uint32_t)sp[0] | ((uint32_t)sp[1] << 8) | ((uint32_t)sp[2] << 16) | ((uint32_t)sp[3] << 24);
        if (lane == 0) {
          st_relaxed_u64(a.status + tile, make_status(epoch, kFlagInclusive, (uint32_t)(excl + agg)));
          yv[lo] = dq(excl);
        }
      } else {
        if (lane == 0) st_relaxed_u64(a.status + tile, make_status(epoch, kFlagAggregate, agg));
        excl = (uint32_t)lookback_sum(a.status, tile, first_tile, epoch, a.err);
        if (lane == 0) st_relaxed_u64(a.status + tile, make_status(epoch, kFlagInclusive, (uint32_t)(excl + agg)));
      }
      if (lane == 0) s_base = excl;
    }
    __syncthreads();
    q0 = s_base + wexcl;
  }

  for (uint32_t k = 0; k < a.bpw; k++) {
    uint32_t bi = wfirst + k;
    if (bi >= dt.nblk) break;
    uint64_t b = dt.blk0 + bi, hp;
    uint64_t s = blk_start(b);
    uint32_t m = blk_len(b);
    hp = 0;
    uint32_t bc = cache ? 0u : blk_hdr(b, m, hp);  // the cache holds the deltas
    if (bc == 255u) {
      corrupt = true;
      bc = 0;
    }
    if (FM2) {
      // blockSize 1: the reference's decoder reads no header byte for a
      // one-value block and so steps 4 bytes per block where its encoder
      // wrote 5 (szpd_float.cc:483, szpd_double.cc:487); results follow it
      const uint64_t so = L == 1 ? R0 + 4 * b : hp - 4;
      if (so + 4 > R1) {
        corrupt = true;
        q0 = 0;
      } else {
        const uint8_t* sp = in + so;
        q0 = (uint32_t)__ldg(sp) | ((uint32_t)__ldg(sp + 1) << 8) | ((uint32_t)__ldg(sp + 2) << 16) |
             ((uint32_t)__ldg(sp + 3) << 24);
      }
      if (lane == 0) yv[s - 1] = dq(q0);
    }
    uint32_t dk = 0;
    if (cache) {
#pragma unroll
      for (int c = 0; c < KC; c++)
        if ((uint32_t)c == k) dk = cd[c];
    }
    for (uint32_t p0 = 0; p0 < m; p0 += 32) {
      uint32_t j = p0 + lane;
      uint32_t d = cache ? dk : ((bc && j < m) ? decode_delta(in + hp, m, bc, j) : 0u);
      uint32_t sc = warp_incl_scan(d, lane);
      if (j < m) yv[s + j] = dq(q0 + sc);
      q0 += __shfl_sync(0xffffffffu, sc, 31);
    }
  }
  if (__any_sync(0xffffffffu, corrupt) && lane == 0) atomicOr(fd.err, kErrCorrupt);
}

cudaError_t launch_dec_setup(const DecArgs& a, cudaStream_t st) {
  dec_setup_kernel<false><<<1, 1024, 0, st>>>(a);  // a field of 0.5 GB has 7000 tickets to write
  return cudaGetLastError();
}

cudaError_t launch_dec_setup_batch(const DecArgs& a, uint32_t nfields, cudaStream_t st) {
  if (nfields == 0) return cudaSuccess;
  dec_setup_kernel<true><<<nfields, 256, 0, st>>>(a);
  return cudaGetLastError();
}

template <bool FM2>
static cudaError_t launch_locate_t(const DecArgs& a, cudaStream_t st) {
  const size_t smem = locate_smem_bytes(a.super_chunk, a.overlap, a.maxsz);
  auto k = locate_packs(a.super_chunk, a.maxsz) ? locate_kernel<FM2, true> : locate_kernel<FM2, false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<a.nlocate_ctas, kLocThreads, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_locate(const DecArgs& a, cudaStream_t st) {
  if (a.nlocate_ctas == 0) return cudaSuccess;
  return a.fm2 ? launch_locate_t<true>(a, st) : launch_locate_t<false>(a, st);
}

uint32_t decode_blocks_per_tile(uint32_t L, uint32_t& bpw) {
  const uint32_t b = 2048u / (L < 32 ? 32u : L);
  bpw = b < 1 ? 1 : (b > 8 ? 8 : b);
  return kDecWarps * bpw;
}

cudaError_t launch_decode_f64(const DecArgs& a, cudaStream_t st) {
  if (a.fm2) {
    decode_generic<kDecWarps, true, double><<<a.ntiles, kDecWarps * 32, 0, st>>>(a);
  } else {
    decode_generic<kDecWarps, false, double><<<a.ntiles, kDecWarps * 32, 0, st>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_decode(const DecArgs& a, cudaStream_t st) {
  if (a.fm2) {
    decode_generic<kDecWarps, true><<<a.ntiles, kDecWarps * 32, 0, st>>>(a);
  } else {
    decode_generic<kDecWarps, false><<<a.ntiles, kDecWarps * 32, 0, st>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace szp
