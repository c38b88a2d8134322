// decode_flow.cu -- the fastmode1 / fastmode2 decoder for blockSize 8..256 (a
// power of two): one kernel from stream bytes to values.
//
// A segment's stream is cut into super-chunks of 1 to 16 KB and each CTA takes
// one at a time, in ticket order:
//
//   stage   one bulk copy brings the super-chunk (and a lead-in before it) to
//           shared memory, where it stays until its values are written
//   walk    the block headers are found.  The stream keeps no index: a block's
//           position depends on every bit count before it in its segment.  The
//           super-chunk is cut into 1 to 16 chunks; the warps first find where the
//           header chain crosses each chunk's start (chains started on payload
//           die, a header byte must be <= 33, or fall in with the true chain), then
//           a lane walks each chunk and notes its blocks.  A lane whose
//           predecessor did not leave where it entered walks again.
//   sum     (fastmode1) all warps unpack the blocks' deltas once, for the sum of
//           each group of 256 values
//   look back  the CTA publishes (block count, delta sum, entry, exit) and sums
//           the predecessors' by a decoupled look-back over the segment, which
//           also checks that the predecessor's exit is this entry; a wrong entry
//           (rare) is corrected and walk and sum run again
//   decode  the base value is now known: each warp unpacks its groups again,
//           scans them in registers, dequantizes and stores them, 32 bytes per
//           lane, with no further exchange between warps
//
// What bounds it: the waits between the steps of a super-chunk.  With 7 CTAs of 4
// warps per SM, issue is 65 % and the ALU 56 % busy, DRAM 30 %; the largest stall is
// the barrier, where three warps wait while one walks (2^26 values at REL 1e-3).
// Why this shape: the pipeline it replaces (a pass that located blocks, 4
// bytes of index per block, a decode that held 32 KB of decoded values per tile
// through a look-back over up to 304 tiles, two CTAs per SM) took 0.094 + 0.256
// ms for a 512^3 field at REL 1e-3; here the bytes held are the compressed
// ones, the stream is read once, and it takes 0.208 ms.  fastmode2, which has no
// sum, went from 0.125 + 0.130 to 0.104 ms for 384^3 values in blocks of 64.
// Measured on the way, for the 512^3 field: a chain step with range checks took
// 170 cycles, one without 55 (0.373 -> 0.316 ms with the branch-free walk); 8
// CTAs of 64 registers spill, 0.26 ms; segments taken one after the other, not
// in turns, 0.373 against 0.291 ms.
#include <atomic>
#include <cstring>
#include <type_traits>

#include "szp_device.cuh"
#include "szp_f64.h"
#include "szp_kernels.h"
#include "szp_pipe.cuh"
#include "szp_tma.cuh"
#include "szp_unpack.cuh"

namespace szp {
namespace {

constexpr int kFlowWarps = 4;
constexpr int kFlowThreads = 32 * kFlowWarps;
constexpr uint32_t kEnd = 0xFFFFFFFEu;   // the walk left the segment region
constexpr uint32_t kDead = 0xFFFFFFFFu;  // the walk met an invalid header

// Shape of the decoder for blocks of 8*LPB values: up to 16 KB of stream per
// CTA, cut into 2 to 16 chunks that hold 7 blocks of the largest size.
template <int LPB>
struct Shape {
  static constexpr uint32_t L = 8 * LPB;
  static constexpr uint32_t BPR = 32 / LPB;                   // blocks per group of 256 values
  static constexpr uint32_t C = LPB <= 4 ? 1024 : 256 * LPB;  // bytes per chunk (a walking lane)
  static constexpr uint32_t CL = LPB <= 4 ? 10 : LPB == 8 ? 11 : LPB == 16 ? 12 : 13;
  static constexpr uint32_t NB = kFlowSuper / C;              // chunks
  static constexpr uint32_t KCAP = LPB <= 4 ? 1536 : LPB == 8 ? 1024 : LPB == 16 ? 768 : 512;  // blocks listed at a time
  static_assert(C == 1u << CL, "chunks of a power of two");
};

// fastmode1 blocks of 8 and 16 values may take little more than a byte each, and
// a lane's walk is a chain of dependent steps: the setup kernel gives them
// chunks of down to C / 8 (flow_shape).  (33.5 M values in blocks of 8 at 0.23
// bytes a value: 0.46 ms with chunks of C, 0.16 so.  For blocks of 32 the
// run-time chunk cost 3 % at ordinary bounds.)
template <int LPB, bool FM2>
constexpr bool kVarChunks = LPB <= 2 && !FM2;
// Bytes walked before a chunk to find its entry: 4 or more of the largest blocks,
// and half of it before shorter chunks of 16-value blocks (always half: more
// wrong entries, 33.5 M values in one segment at 1.33 bytes a value 115 -> 176 us;
// never: 134 M values at 0.09 bytes a value 441 -> 597 us).
template <int LPB>
constexpr uint32_t kWindow = LPB == 1 ? 128 : Shape<LPB>::C / 2;
template <int LPB, bool FM2>
constexpr uint32_t kLead = FM2 ? 4096 : kWindow<LPB>;  // bytes staged before a super-chunk
// Runs of empty blocks that the walking lanes note (134 M values in blocks of 8 at
// 0.18 bytes a value, where 128 are too few: 719 -> 660 us).
template <int LPB, bool FM2>
constexpr uint32_t kRuns = kVarChunks<LPB, FM2> ? 256 : 128;

template <int LPB, bool FM2>
__host__ __device__ constexpr uint32_t flow_maxsz() {
  // bit count 33: 4 byte planes and one remainder bit per value
  constexpr uint32_t L = 8 * LPB, m = FM2 ? L - 1 : L;
  return 1 + (m + 7) / 8 + 4 * m + (m + 7) / 8 + (FM2 ? 4 : 0);
}

// Bytes of the staging buffer: a lead-in and a super-chunk from any 16-byte
// phase, the last block's rest, and what loads read past a block's end.
template <int LPB, bool FM2>
__host__ __device__ constexpr uint32_t flow_smem() {
  return 16 + kLead<LPB, FM2> + kFlowSuper + flow_maxsz<LPB, FM2>() + 8 + 32;
}

// The super-chunk a CTA is working on.
struct FlowTile {
  uint64_t nb;     // blocks of the segment
  uint64_t lo, hi; // its elements
  void* y;         // the field's output
  uint32_t* err;   // the field's error word
  double ebd;
  float eb;
  uint32_t tile, j, rec, last;  // ticket; position in the segment; look-back record; whether it is the last
  uint32_t strict;          // another segment follows: the region holds the segment's blocks and no more
  uint32_t sc;              // bytes of the segment's super-chunks
  uint32_t cl;              // log2 of their chunks' bytes
  uint32_t scS, scE, rlen;  // region offsets of the super-chunk and the region's length
  uint32_t st0, st1;        // region offsets of the staged bytes
  uint32_t align;           // shared-memory offset of the first staged byte
  uint32_t seed;            // q of the segment's first element (fastmode1, j == 0)
  uint32_t hb0, hb1, tb0, tb1;  // shared-memory offsets staged by plain loads
};

// What a warp found in its window of a look-back.
struct FlowWindow {
  uint32_t state;  // 0 all aggregates, 1 not ready for too long, 2 a broken chain, 3 ends at an inclusive record
  uint32_t cnt, sum;
  uint32_t exit, entry;  // of the nearest tile, of the farthest
};

// One look-back record: two words, each tagged with epoch and flag; a record is
// read when both tags agree.  The 42-bit values hold
//   first   aggregate: entry (16, from the super-chunk's start), count (16), exit low bits (10)
//           inclusive: count before and with the super-chunk (32), exit low bits (10)
//   second  delta sum (32), exit high bits (10)
// with the exit counted from the super-chunk's end.
constexpr uint32_t kHDead = 0xFFFFu, kHEnd = 0xFFFEu, kXDead = 0xFFFu, kXEnd = 0xFFEu;

// an aggregate for a super-chunk's second entry (a tag of its own, so that no read record mixes two)
constexpr uint64_t kFlagSecond = 0;
__device__ __forceinline__ void publish(uint64_t* st, uint32_t epoch, uint64_t flag, uint64_t cnt, uint32_t sum,
                                        uint32_t h, uint32_t x, uint32_t scS, uint32_t scE) {
  const uint32_t xr = x == kDead ? kXDead : x == kEnd ? kXEnd : x - scE;
  const uint32_t hr = h == kDead ? kHDead : h == kEnd ? kHEnd : h - scS;
  const uint64_t head = flag != kFlagInclusive ? ((uint64_t)hr << 16 | cnt) : cnt;
  st_relaxed_u64(st, make_status(epoch, flag, head << 10 | (xr & 1023u)));
  st_relaxed_u64(st + 1, make_status(epoch, flag, (uint64_t)sum << 10 | (xr >> 10)));
}

__device__ __forceinline__ ulonglong2 ld_record(const uint64_t* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}

// What an invalid header adds to a chain's position: more than any offset, and
// little enough that a chain that goes on stepping there does not wrap around.
constexpr uint32_t kAway = 1u << 17;

// Header chains over the staged bytes; positions are shared-memory offsets.
template <int LPB, bool FM2>
struct Chain {
  const uint8_t* s;
  uint32_t avail;  // bytes are staged below this offset
  uint32_t last;   // the last offset a header may be read at (the end of the buffer)
  // One block on from p; b receives its bit count.  A walk is a chain of these
  // dependent steps, so there is no predicate and no branch in it (55 cycles a
  // step; one with range checks took 170): an invalid header sends the chain
  // beyond any offset for good, and offsets out of the buffer read its last byte.
  __device__ __forceinline__ uint32_t next(uint32_t p, uint32_t& b) const {
    b = s[min(p, last) + (FM2 ? 4 : 0)];
    const uint32_t bad = (uint32_t)((int32_t)(kMaxBitCount - b) >> 31) & kAway;
    if (FM2) {
      constexpr uint32_t M = 8 * LPB - 1;
      const uint32_t out = (uint32_t)((int32_t)(avail - 5 - p) >> 31) & kAway;  // the header byte is not staged
      return p + out + (5 + LPB * min(b, 1u) + (b >> 3) * M + (((b & 7) * M + 7) >> 3)) + bad;
    }
    return p + (1 + LPB * b) + (LPB * min(b, 1u) + bad);
  }
  // over a run of empty blocks from p (a zero byte each; fastmode2: five, the
  // seed of a field that is 0 and the bit count), up to lim; k counts them
  __device__ __forceinline__ void zeros(uint32_t& p, uint32_t lim, uint32_t& k) const {
    constexpr uint32_t E = kEmpty;
    const uint32_t stop = FM2 ? min(lim + E, avail) : lim;
    uint32_t z = p;  // the first byte that is not zero
    while (z < stop) {
      if ((z & 15) == 0 && z + 16 <= stop) {
        const uint4 v = *reinterpret_cast<const uint4*>(s + z);
        if ((v.x | v.y | v.z | v.w) == 0) {
          z += 16;
          continue;
        }
      }
      const uint32_t left = 4 - (z & 3);
      const uint32_t w = *reinterpret_cast<const uint32_t*>(s + (z & ~3u)) >> (8 * (z & 3));
      const uint32_t n = min(min(w ? (uint32_t)(__ffs(w) - 1) >> 3 : left, left), stop - z);
      z += n;
      if (n < left) break;
    }
    uint32_t n = z - p;
    if (FM2) n = p < lim ? min(n / E, (lim - p + E - 1) / E) : 0u;
    p += n * E;
    k += n;
  }
  static constexpr uint32_t kEmpty = FM2 ? 5 : 1;  // bytes of an empty block
};

// ------------------------------------------------------------------ output --
template <int OUT>
struct Elem {
  using T = float;
};
template <>
struct Elem<kOutDouble> {
  using T = unsigned long long;  // doubles, written as their bits
};

// (float)q * eb, the code itself, or the code added to the one in place.
template <int OUT>
struct Put {
  float eb;
  DequantD dd;
  bool rare;  // a bound whose products need the x86 NaN rule, or (float64) the FP64 multiply
  bool wrap = false;
  __device__ __forceinline__ Put(float e, double ed) : eb(e), dd(OUT == kOutDouble ? ed : 1.0) {
    rare = OUT == kOutFloat ? !isfinite(e) : OUT == kOutDouble && !dd.fast;
  }
  // not for a rare bound
  __device__ __forceinline__ float value(uint32_t q) const {
    return OUT >= kOutCodes ? __uint_as_float(q) : dequant(q, eb);
  }
  // Of a lane's 8 doubles, three take the FP64 pipe, which is otherwise idle
  // (2 lanes a clock and SM), and five the integer arithmetic that bounds the
  // kernel; both round as binary64 does (33.5 M doubles: 214 us all integer,
  // 182 so).
  template <int J>
  __device__ __forceinline__ unsigned long long value_d(uint32_t q) const {
    if (J == 1 || J == 4 || J == 6) return (unsigned long long)__double_as_longlong(__dmul_rn((double)(int32_t)q, dd.eb));
    return f64i::dequant_bits((int32_t)q, dd.m, dd.ef, dd.sgn);
  }
  __device__ __forceinline__ float add(float old, uint32_t q) {  // old + q as int32 codes
    const int32_t x = (int32_t)__float_as_uint(old), y = (int32_t)q;
    const int32_t z = (int32_t)((uint32_t)x + (uint32_t)y);
    wrap |= ((x ^ z) & (y ^ z)) < 0;
    return __uint_as_float((uint32_t)z);
  }
  // one element, any bound
  __device__ __forceinline__ void one(void* y, uint64_t e, uint32_t q) {
    if (OUT == kOutDouble) {
      static_cast<unsigned long long*>(y)[e] = dd(q);
    } else {
      float* p = static_cast<float*>(y) + e;
      *p = OUT == kOutCodesAdd ? add(*p, q) : OUT == kOutCodes ? value(q) : dequant(q, eb, rare);
    }
  }
};

// 8 values at a 32-byte-aligned address (64 bytes of doubles).
template <int OUT>
__device__ __forceinline__ void store8(Put<OUT>& put, void* dst, const uint32_t (&q)[8]) {
  if constexpr (OUT == kOutDouble) {
    unsigned long long* p = static_cast<unsigned long long*>(dst);
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(put.template value_d<0>(q[0])),
                 "l"(put.template value_d<1>(q[1])), "l"(put.template value_d<2>(q[2])),
                 "l"(put.template value_d<3>(q[3]))
                 : "memory");
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p + 4), "l"(put.template value_d<4>(q[4])),
                 "l"(put.template value_d<5>(q[5])), "l"(put.template value_d<6>(q[6])),
                 "l"(put.template value_d<7>(q[7]))
                 : "memory");
  } else {
    float v[8];
    if constexpr (OUT == kOutCodesAdd) {
      asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                   : "l"(dst)
                   : "memory");
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = put.add(v[j], q[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = put.value(q[j]);
    }
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(v[0]), "f"(v[1]),
                 "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
  }
}

// Two groups' values, one after the other from dst (element 8l + j of the first
// group in lane l, V of the 64 lanes hold values), where dst is SH elements
// past a 32-byte boundary (SH > 0) or -SH before one: every lane passes its
// last SH (takes the next lane's first -SH) values on, so that all but the ends
// of the run go out as aligned 32-byte stores.  (Through shared memory and
// 16-byte stores the same took two and a half times the instructions.)
template <int OUT, int SH, typename E>
__device__ __forceinline__ void store_shifted(Put<OUT>& put, E* dst, const uint32_t (&q)[2][8], uint32_t V, int lane) {
  constexpr int N = SH > 0 ? SH : -SH;
  const int from = SH > 0 ? (lane + 31) & 31 : (lane + 1) & 31;
  uint32_t c[2][N];
#pragma unroll
  for (int u = 0; u < 2; u++)
#pragma unroll
    for (int j = 0; j < N; j++) c[u][j] = __shfl_sync(0xffffffffu, q[u][SH > 0 ? 8 - N + j : j], from);
#pragma unroll
  for (int u = 0; u < 2; u++) {
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if constexpr (SH > 0) {
        o[j] = j >= N ? q[u][j - N] : u && lane == 0 ? c[0][j] : c[u][j];
      } else {
        o[j] = j < 8 - N ? q[u][j + N] : u == 0 && lane == 31 ? c[1][j + N - 8] : c[u][j + N - 8];
      }
    }
    const uint32_t at = 32 * u + lane;
    if (SH > 0 ? at > 0 && at < V : at + 1 < V) store8<OUT>(put, dst + 8 * at - SH, o);
  }
  if (lane == 0 && V) {  // the first lane's values before the first whole 32 bytes
#pragma unroll
    for (int j = 0; j < (SH > 0 ? 8 - N : N); j++) put.one(dst, j, q[0][j]);
  }
  if (V && lane == (int)((V - 1) & 31)) {  // the last lane's after the last
#pragma unroll
    for (int j = SH > 0 ? 8 - N : N; j < 8; j++) put.one(dst, 8 * (V - 1) + j, V > 32 ? q[1][j] : q[0][j]);
  }
}

// o[u][j] = the value SH elements before (SH > 0) or -SH after element
// 32*8u + 8*lane + j of the two groups' values q.
template <int SH>
__device__ __forceinline__ void shift_groups(uint32_t (&o)[2][8], const uint32_t (&q)[2][8], int lane) {
  constexpr int N = SH > 0 ? SH : -SH;
  const int from = SH > 0 ? (lane + 31) & 31 : (lane + 1) & 31;
  uint32_t c[2][N];
#pragma unroll
  for (int u = 0; u < 2; u++)
#pragma unroll
    for (int j = 0; j < N; j++) c[u][j] = __shfl_sync(0xffffffffu, q[u][SH > 0 ? 8 - N + j : j], from);
#pragma unroll
  for (int u = 0; u < 2; u++) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if constexpr (SH > 0) {
        o[u][j] = j >= N ? q[u][j - N] : u && lane == 0 ? c[0][j] : c[u][j];
      } else {
        o[u][j] = j < 8 - N ? q[u][j + N] : u == 0 && lane == 31 ? c[1][j + N - 8] : c[u][j + N - 8];
      }
    }
  }
}

// store_shifted for doubles, whose conversion is too long to have one copy of it
// for each shift and each end: the ends go through `ends` (16 words of shared
// memory), one element per lane.  (For floats the seven copies are the faster:
// 232 us against 238 on 134 M values.)
__device__ __forceinline__ void store_doubles(Put<kOutDouble>& put, unsigned long long* dst, const uint32_t (&q)[2][8], uint32_t V,
                                              int sh, int lane, uint32_t* ends) {
  __syncwarp();
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < 8; j++) ends[j] = q[0][j];
  }
  if (V && lane == (int)((V - 1) & 31)) {
#pragma unroll
    for (int j = 0; j < 8; j++) ends[8 + j] = V > 32 ? q[1][j] : q[0][j];
  }
  __syncwarp();
  if (V && lane < 16) {
    // the first lane's values before the first whole 64 bytes, the last lane's after the last
    const int j = lane & 7, head = sh > 0 ? 8 - sh : -sh;
    if (lane < 8 ? j < head : j >= head) put.one(dst, (lane < 8 ? 0 : 8 * (V - 1)) + j, ends[lane]);
  }
  uint32_t o[2][8];
  switch (sh) {
    case 1: shift_groups<1>(o, q, lane); break;
    case 2: shift_groups<2>(o, q, lane); break;
    default: shift_groups<-1>(o, q, lane); break;
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const uint32_t at = 32 * u + lane;
    if (sh > 0 ? at > 0 && at < V : at + 1 < V) store8<kOutDouble>(put, dst + 8 * (int)at - sh, o[u]);
  }
}

template <int OUT, typename E>
__device__ __forceinline__ void store_groups(Put<OUT>& put, E* dst, const uint32_t (&q)[2][8], uint32_t V, int lane,
                                             uint32_t* ends) {
  constexpr uint32_t U = 32 / sizeof(E);  // elements in 32 bytes
  const uint32_t s = (uint32_t)((uintptr_t)dst / sizeof(E)) % U;
  if (put.rare) {
#pragma unroll 1
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (32u * u + lane < V) put.one(dst, 256 * u + 8 * lane + j, u ? q[1][j] : q[0][j]);
    return;
  }
  if (s == 0) {
#pragma unroll
    for (int u = 0; u < 2; u++)
      if (32u * u + lane < V) store8<OUT>(put, dst + 256 * u + 8 * lane, q[u]);
    return;
  }
  if constexpr (OUT == kOutDouble) {
    store_doubles(put, dst, q, V, s == 3 ? -1 : (int)s, lane, ends);
  } else {
    switch (s) {
      case 1: store_shifted<OUT, 1>(put, dst, q, V, lane); break;
      case 2: store_shifted<OUT, 2>(put, dst, q, V, lane); break;
      case 3: store_shifted<OUT, 3>(put, dst, q, V, lane); break;
      case 4: store_shifted<OUT, 4>(put, dst, q, V, lane); break;
      case 5: store_shifted<OUT, -3>(put, dst, q, V, lane); break;
      case 6: store_shifted<OUT, -2>(put, dst, q, V, lane); break;
      default: store_shifted<OUT, -1>(put, dst, q, V, lane); break;
    }
  }
}

// Lists blocks [kb, kb + cap) of a super-chunk whose blocks are more than the list
// holds, from what the walking lanes noted of its 1 << lg chunks: the blocks between
// a chunk's runs of empty ones (E bytes each), and the runs.  All threads.
// Out of line: few super-chunks come here, and inlined it cost every other 3 %.
static __device__ __noinline__ void gather_window(uint16_t* pos, const uint16_t* note, const uint32_t* notes,
                                                  const uint32_t* runs, const uint16_t* lens, const uint32_t* c0s,
                                                  uint32_t note_share, uint32_t run_share, uint32_t lg, uint32_t kb,
                                                  uint32_t cap, uint32_t E) {
  const uint32_t tid = threadIdx.x, TPC = kFlowThreads >> lg, i = tid / TPC, first = tid & (TPC - 1);  // threads per chunk
  const uint32_t c0 = c0s[i], n = c0s[i + 1] - c0;
  const uint32_t nn = n ? notes[i] & 0xFFFFu : 0u, nruns = n ? notes[i] >> 16 : 0u;
  uint32_t t0 = 0, at = c0 - kb;  // the next note, and its place in the list (before the list: wraps around)
  for (uint32_t g = 0; g <= nruns; g++) {
    const uint32_t run = g < nruns ? runs[i * run_share + g] : nn << 16, len = g < nruns ? lens[i * run_share + g] : 0u;
    const uint32_t t1 = run >> 16;
    for (uint32_t t = t0 + first; t < t1; t += TPC)
      if (at + t - t0 < cap) pos[at + t - t0] = note[i * note_share + t];
    at += t1 - t0;
    for (uint32_t t = first; t < len; t += TPC)
      if (at + t < cap) pos[at + t] = (uint16_t)((run & 0xFFFFu) + t * E);
    at += len;
    t0 = t1;
  }
}

template <int LPB, bool BATCH, bool FM2, int OUT>
__global__ void __launch_bounds__(kFlowThreads, 7) decode_flow(const __grid_constant__ DecArgs a) {
  using S = Shape<LPB>;
  constexpr uint32_t L = S::L, BPR = S::BPR, KCAP = S::KCAP, MAXSZ = flow_maxsz<LPB, FM2>();
  constexpr uint32_t NB = S::NB, WIN = kWindow<LPB>, NOTES = kFlowNotes, RUNS = kRuns<LPB, FM2>;
  extern __shared__ __align__(16) uint8_t s_b[];
  __shared__ uint16_t s_pos[KCAP];          // headers of the listed blocks (shared-memory offsets)
  __shared__ uint32_t s_tot[KCAP / BPR + 1];  // delta sums of the groups, then their exclusive prefixes
  __shared__ uint16_t s_note[NOTES + 32];  // the blocks that walking lanes note
  // and the runs of empty blocks they took at once: notes before << 16 | first offset; length
  __shared__ uint32_t s_runs[RUNS];
  __shared__ uint16_t s_len[RUNS];
  __shared__ uint32_t s_notes[NB];    // notes | runs << 16
  __shared__ uint32_t s_tried[kFlowWarps][32];
  __shared__ uint32_t s_ent[NB];            // entries of the chunks (shared-memory offsets, kDead: none found)
  __shared__ uint32_t s_c0[NB + 1];         // blocks before each chunk
  __shared__ bool s_noted, s_many;          // the walking lanes noted every block and run; and there are more than KCAP
  __shared__ FlowTile s_t;
  __shared__ uint32_t s_k, s_sum, s_h0, s_epoch;
  __shared__ FlowWindow s_win[kFlowWarps];
  __shared__ __align__(8) uint64_t s_bar;
  if (!BATCH) wait_for_previous();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sub = lane % LPB, grp = lane / LPB;
  uint32_t epoch = 0;
  const uint32_t total = *a.ticket_total;
  if (tid == 0) {
    mbar_init(&s_bar, 1);
    epoch = *(volatile uint32_t*)&a.ls->epoch;
    s_epoch = epoch;
    __threadfence();
  }
  epoch = __shfl_sync(0xffffffffu, epoch, 0);  // used by warp 0 only
  uint32_t parity = 0;
  for (;;) {
    __syncthreads();  // every read of the tile before is done
    if (tid == 0) {
      const uint32_t tile = draw_ticket_persistent(a.ls, total);
      s_t.tile = tile;
      if (tile < total) {
        const uint4 at = a.map[tile];  // field, segment, position in it and shape, look-back record
        const DecField& fd = BATCH ? a.fields[at.x] : a.f;
        const Segments sg = fd.seg;
        const uint64_t R0 = fd.reg0[at.y], R1 = fd.reg1[at.y];
        FlowTile t;
        t.tile = tile;
        t.j = at.z & kFlowPosMask;
        t.rec = at.w;
        t.strict = at.y + 1 < sg.T;
        t.rlen = (uint32_t)(R1 - R0);
        const uint32_t shape = at.z >> kFlowPosBits;
        t.cl = S::CL - (kVarChunks<LPB, FM2> ? shape >> 4 : 0u);
        t.sc = ((shape & 15) + 1) << t.cl;
        t.scS = t.j * t.sc;
        t.scE = t.scS + min(t.sc, t.rlen - t.scS);  // (a region may end a byte below 4 GiB)
        t.last = t.scE == t.rlen;
        const uint32_t lead = min(kLead<LPB, FM2>, a.overlap);
        t.st0 = t.scS > lead ? t.scS - lead : 0u;
        t.st1 = (uint32_t)min((uint64_t)t.rlen, (uint64_t)t.scE + MAXSZ + 8);
        // the 16-byte-aligned part of the staged bytes that lies in the stream goes by bulk copy
        const uintptr_t in = (uintptr_t)fd.in, g0 = in + R0 + t.st0, g1 = in + R0 + t.st1;
        const uintptr_t a0 = g0 & ~(uintptr_t)15;
        const uintptr_t b0 = max(a0, (in + 15) & ~(uintptr_t)15);
        const uintptr_t b1 = min((g1 + 15) & ~(uintptr_t)15, (in + fd.len) & ~(uintptr_t)15);
        t.align = (uint32_t)(g0 - a0);
        const uint32_t end = t.align + (t.st1 - t.st0);
        t.hb0 = t.align;
        t.tb1 = end;
        if (b1 > b0) {
          t.hb1 = min(max((uint32_t)(b0 - a0), t.align), end);
          t.tb0 = max(min((uint32_t)(b1 - a0), end), t.hb1);
          fence_async_smem();
          mbar_arrive_expect_tx(&s_bar, (uint32_t)(b1 - b0));
          bulk_load(s_b + (b0 - a0), reinterpret_cast<const void*>(b0), (uint32_t)(b1 - b0), &s_bar);
        } else {
          t.hb1 = end;
          t.tb0 = end;
          mbar_arrive(&s_bar);
        }
        t.lo = sg.lo(at.y);
        t.hi = sg.hi(at.y);
        t.nb = FM2 ? (t.hi - t.lo + L - 1) / L : (t.hi - t.lo > 1 ? (t.hi - t.lo - 1 + L - 1) / L : 0);
        t.y = fd.y;
        t.err = fd.err;
        t.eb = fd.plan->eb;
        t.ebd = fd.plan->ebd;
        t.seed = 0;
        if (!FM2 && t.j == 0) {
          const uint8_t* sp = fd.in + R0 - 4;  // the segment's 4-byte seed precedes its blocks
          t.seed = (uint32_t)__ldg(sp) | ((uint32_t)__ldg(sp + 1) << 8) | ((uint32_t)__ldg(sp + 2) << 16) |
                   ((uint32_t)__ldg(sp + 3) << 24);
        }
        s_t = t;
        // the ragged ends, which only the stream's own start and end have
        const uint8_t* g = reinterpret_cast<const uint8_t*>(a0);
        for (uint32_t b = t.hb0; b < t.hb1; b++) s_b[b] = __ldg(g + b);
        for (uint32_t b = t.tb0; b < t.tb1; b++) s_b[b] = __ldg(g + b);
      }
    }
    __syncthreads();
    const uint32_t tile = s_t.tile;
    if (tile >= total) return;
    if (!mbar_wait_ns(&s_bar, parity, kWaitNs)) {
      atomicOr(a.err, kErrLookbackTimeout);
      mbar_wait_ns(&s_bar, parity, kWaitNs);  // the copy lands before the CTA goes on or exits
    }
    parity ^= 1;

    const uint32_t off = s_t.align - s_t.st0;  // region offset p is at s_b[p + off]
    const Chain<LPB, FM2> ch{s_b, s_t.st1 + off, flow_smem<LPB, FM2>() - 8};
    const uint32_t scS = s_t.scS, scE = s_t.scE, rlen = s_t.rlen;
    const bool j0 = s_t.j == 0;
    const uint32_t cl = kVarChunks<LPB, FM2> ? s_t.cl : S::CL;  // log2 of a chunk's bytes

    // ---- entries: where the header chain crosses each chunk's start ----
    // 32 lanes walk from 32 neighbouring bytes, WIN or less before the chunk.  Chains that
    // began on payload meet an invalid header or fall in with the true one; the
    // position that most of them reach is taken (a wrong one is corrected below;
    // 2 in 1000 are, of a walk at REL 1e-3).  Where all die (blocks longer than 32
    // bytes), the next 32 bytes are tried.  A warp does its NB / 4 chunks side by
    // side, after three steps with 8 lanes a chunk.
    const uint32_t lS = scS + off, lE = scE + off;  // the super-chunk in shared-memory offsets
    {
      constexpr int Q = NB >= kFlowWarps ? NB / kFlowWarps : 1;
      uint32_t at[Q], p[Q];  // first byte tried; the lane's position
      uint32_t back[Q];      // the window
      uint32_t open = 0;     // chunks without an entry yet
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const uint32_t i = warp + kFlowWarps * q, B = lS + (i << cl);
        const uint32_t first = s_t.st0 + off;
        back[q] = WIN >> (kVarChunks<LPB, FM2> && LPB == 2 && cl < S::CL);
        at[q] = B - first > back[q] ? B - back[q] : first;
        p[q] = kAway;
        if (i < NB && B < lE && !(i == 0 && j0)) {
          open |= 1u << q;
          p[q] = at[q] + lane;
        }
        if (i < NB && lane == 0) s_ent[i] = kDead;
      }
      // A run of zero bytes longer than the largest block holds a header, and every
      // byte from there to the run's end is an empty block: the chain passes
      // the byte after the last such run before the chunk (16 bytes per lane).
      if constexpr (!FM2 && LPB <= 8) {
        constexpr int R = (MAXSZ + 15) / 16;
#pragma unroll
        for (int q = 0; q < Q; q++) {
          if (!(open >> q & 1)) continue;
          const uint32_t B = lS + ((warp + kFlowWarps * q) << cl), g = (B & ~15u) - 512 + 16 * lane;
          const bool in = (int32_t)g >= (int32_t)at[q];
          const uint4 v = in ? *reinterpret_cast<const uint4*>(s_b + g) : make_uint4(1, 0, 0, 0);
          uint32_t m = __ballot_sync(0xffffffffu, (v.x | v.y | v.z | v.w) == 0);
#pragma unroll
          for (int len = 1; len < R;) {  // m: last lanes of runs of `len` lanes
            const int sft = len < R - len ? len : R - len;
            m &= m << sft;
            len += sft;
          }
          if (m) p[q] = (B & ~15u) - 512 + 16 * (32 - __clz(m));
        }
      }
      uint32_t* tried = s_tried[warp];  // the survivors of a chunk, 8 places each
      while (open) {
        // three steps from 32 bytes of each chunk; most chains that began on payload die here
        uint32_t b, past[Q];  // past: how far past the chunk's start its chain crosses it
#pragma unroll
        for (int q = 0; q < Q; q++) past[q] = p[q] - (lS + ((warp + kFlowWarps * q) << cl));
#pragma unroll
        for (int u = 0; u < 3; u++)
#pragma unroll
          for (int q = 0; q < Q; q++) {
            p[q] = ch.next(p[q], b);
            past[q] = min(past[q], p[q] - (lS + ((warp + kFlowWarps * q) << cl)));  // the first past it: the smallest
          }
        __syncwarp();
        if (lane < 8 * Q) tried[lane] = kAway;
        __syncwarp();
#pragma unroll
        for (int q = 0; q < Q; q++) {
          const uint32_t B = lS + ((warp + kFlowWarps * q) << cl);
          const bool alive = (p[q] < kAway || past[q] <= MAXSZ) && at[q] + lane < B;
          const uint32_t m = __ballot_sync(0xffffffffu, alive), n = __popc(m & ((1u << lane) - 1u));
          if (alive && n < 8) tried[8 * q + n] = past[q] <= MAXSZ ? B + past[q] : p[q];
        }
        __syncwarp();
        // lanes 8q .. 8q + 7: the first 8 survivors of chunk q, on to its start
        const uint32_t B = lS + ((warp + kFlowWarps * min((uint32_t)lane >> 3, (uint32_t)Q - 1)) << cl);
        uint32_t c = lane < 8 * Q ? tried[lane] : kAway, over = c - B;
        bool busy = c < B;
        while (__any_sync(0xffffffffu, busy)) {
          const uint32_t c0 = c;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            c = ch.next(c, b);
            over = min(over, c - B);
          }
          if (c - c0 == 4 * Chain<LPB, FM2>::kEmpty && c < B) {  // a run of empty blocks
            uint32_t k = 0;
            ch.zeros(c, B, k);
            over = min(over, c - B);
          }
          busy = c < B;
        }
        // the crossing that most survivors of a chunk agree on
        const bool alive = over <= MAXSZ;
        const uint32_t e = B + over;
        const uint32_t with = __popc(__match_any_sync(0xffffffffu, alive ? e : kDead));
        uint32_t best = alive ? with << 5 | (31 - lane) : 0u;
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, s));
        const uint32_t ent = __shfl_sync(0xffffffffu, e, 31 - (best & 31));
        uint32_t found = __ballot_sync(0xffffffffu, best != 0 && (lane & 7) == 0);
        // fastmode2: a run of empty blocks has five chains that all stay valid, and
        // only what lies before it tells them apart: where survivors disagree, a
        // window four times as long is tried, as far as there are bytes
        const uint32_t split = FM2 ? __ballot_sync(0xffffffffu, alive && with < best >> 5 || alive && e != ent) : 0u;
        if (best != 0 && (lane & 7) == 0 && (open >> (lane >> 3) & 1)) s_ent[warp + kFlowWarps * (lane >> 3)] = ent;
#pragma unroll
        for (int q = 0; q < Q; q++) {
          p[q] = kAway;
          if (!(open >> q & 1)) continue;
          if (FM2 && (split >> (8 * q) & 0xFFu)) {
            const uint32_t first = s_t.st0 + off, Bq = lS + ((warp + kFlowWarps * q) << cl);
            if (Bq - first > back[q]) {
              back[q] *= 4;
              at[q] = Bq - first > back[q] ? Bq - back[q] : first;
              p[q] = at[q] + lane;
              continue;
            }
          }
          at[q] += 32;
          if ((found >> (8 * q) & 1) || at[q] >= lS + ((warp + kFlowWarps * q) << cl)) {
            open &= ~(1u << q);
          } else {
            p[q] = at[q] + lane;
          }
        }
      }
    }
    __syncthreads();

    // ---- walk: warp 0, a chunk per lane, from its entry ----
    // the chunks share the room for notes (a super-chunk of mostly empty blocks has
    // few chunks with many blocks each: 2^26 values of a walk at REL 1e-3, where
    // 128 notes a chunk were too few, 300 -> 154 us; a mixed batch 530 -> 461; an
    // 8192^2 field of runs pays for the run-time strides, 222 -> 231)
    const uint32_t lg = 32 - __clz((lE - lS - 1) >> cl);  // 1 << lg chunks at least
    // region position of a shared-memory offset, kEnd past the region
    auto reg = [&](uint32_t p) -> uint32_t { return p - off >= rlen ? kEnd : p - off; };
    const uint32_t cS = lS + (min((uint32_t)lane, NB) << cl), cE = min(cS + (1u << cl), lE);
    const bool act = warp == 0 && lane < (int)NB && cS < cE;
    // the super-chunk's entry (region position); a segment's block region starts with a header
    uint32_t h0 = 0, e0 = kDead;
    if (warp == 0) {
      const uint32_t e = act ? s_ent[lane] : kDead;
      e0 = e == kDead ? kDead : reg(e);
      h0 = j0 ? 0u : __shfl_sync(0xffffffffu, e0, 0);
    }
    uint32_t K = 0, sum = 0, xl = kDead;  // blocks, delta sum and exit of the super-chunk (warp 0)
    uint32_t wp = 0, wi = 0, wn = 0, wp0 = 0, wi0 = 0;  // a lane's place in the list of blocks
    bool repaired = false;
    // lists blocks [kb, kb + KCAP) of the super-chunk (warp 0, in order)
    auto list = [&](uint32_t kb) {
      const uint32_t stop = min(wn, kb + KCAP);
      while (__any_sync(0xffffffffu, wi < stop)) {
        const bool in = wi < stop;
        uint32_t b;
        const uint32_t n = ch.next(in ? wp : lS, b);
        if (in) {
          s_pos[wi - kb] = (uint16_t)wp;
          wi++;
          wp = n;
        }
        // a lane in a run of empty blocks: the whole warp lists it, 512 bytes at a time
        uint32_t zr = FM2 ? 0u : __ballot_sync(0xffffffffu, in && b == 0 && s_b[n] == 0 && wi < stop);
        while (zr) {
          const int src = __ffs(zr) - 1;
          zr &= zr - 1;
          uint32_t P = __shfl_sync(0xffffffffu, wp, src), I = __shfl_sync(0xffffffffu, wi, src);
          const uint32_t lim = __shfl_sync(0xffffffffu, stop, src);
          for (;;) {
            // zero bytes from P in each lane's 16 bytes
            const uint32_t g = (P & ~15u) + 16 * lane, lo = lane ? g : P;
            const bool st = g < ch.avail;
            const uint4 v = st ? *reinterpret_cast<const uint4*>(s_b + g) : make_uint4(1, 1, 1, 1);
            const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
            uint32_t first = g + 16;  // first nonzero byte at or after lo
#pragma unroll
            for (int c = 3; c >= 0; c--) {
              const uint32_t a0 = g + 4 * c;
              const uint32_t w = lo > a0 ? (lo >= a0 + 4 ? 0u : vw[c] >> (8 * (lo - a0)) << (8 * (lo - a0))) : vw[c];
              if (w) first = a0 + ((uint32_t)(__ffs(w) - 1) >> 3);
            }
            const uint32_t stopped = __ballot_sync(0xffffffffu, first < g + 16);
            const int l1 = stopped ? __ffs(stopped) - 1 : 31;
            uint32_t end = __shfl_sync(0xffffffffu, first, l1);
            end = min(end, P + (lim - I));
            for (uint32_t t = P + lane; t < end; t += 32) s_pos[I - kb + (t - P)] = (uint16_t)t;
            I += end - P;
            const bool more = !stopped && I < lim;
            P = end;
            if (!more) break;
          }
          if (lane == src) {
            wp = P;
            wi = I;
          }
        }
      }
    };
    // the delta sums of the kn listed blocks' groups, and their prefixes; all warps
    auto sums = [&](uint32_t kn) -> uint32_t {
      uint32_t run = 0;
      if constexpr (!FM2) {
      // two groups at a time: their loads and votes are in flight together
      for (uint32_t r = warp; r * BPR < kn; r += 2 * kFlowWarps) {
        uint32_t o[2], bc[2], sm[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const uint32_t blk = (r + u * kFlowWarps) * BPR + grp;
          o[u] = blk < kn ? s_pos[blk] : 0u;
          bc[u] = blk < kn ? s_b[o[u]] : 0u;
        }
        const uint32_t top = __reduce_max_sync(0xffffffffu, max(bc[0], bc[1]));
        sm[0] = sm[1] = 0;
        auto sum = [&](auto planes) {
#pragma unroll
          for (int u = 0; u < 2; u++) sm[u] = Deltas<LPB, FM2, decltype(planes)::value>(s_b, o[u], bc[u], sub).total;
        };
        if (top == 0) {  // empty blocks
        } else if (top < 8) {  // the largest bit count: no byte plane, one, two, any
          sum(std::integral_constant<int, 0>{});
        } else if (top < 16) {
          sum(std::integral_constant<int, 1>{});
        } else if (top < 24) {
          sum(std::integral_constant<int, 2>{});
        } else {
          sum(std::integral_constant<int, 3>{});
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          if (top) sm[u] = __reduce_add_sync(0xffffffffu, sm[u]);
          if (lane == 0 && (r + u * kFlowWarps) * BPR < kn) s_tot[r + u * kFlowWarps] = sm[u];
        }
      }
      __syncthreads();
      if (warp == 0) {
        const uint32_t nr = (kn + BPR - 1) / BPR;
        for (uint32_t r0 = 0; r0 < nr; r0 += 32) {
          const uint32_t v = r0 + lane < nr ? s_tot[r0 + lane] : 0u;
          const uint32_t incl = warp_incl_scan(v, lane);
          if (r0 + lane < nr) s_tot[r0 + lane] = run + incl - v;
          run += __shfl_sync(0xffffffffu, incl, 31);
        }
      }
      }
      return run;  // warp 0: the listed blocks' delta sum
    };
    uint64_t cnt0 = 0;  // blocks before the super-chunk, and the value there (in every thread)
    uint32_t base = 0;
    bool known = j0;  // the entry is the true one, and cnt0 and base are known
    uint64_t kind = kFlagAggregate;
    while (true) {
      if (warp == 0) {
        uint32_t e = lane == 0 ? h0 : e0, k = 0, x = kDead;
        bool need = act, noted = true;
        uint32_t differ;
        do {
          const bool go = need && e != kDead && e != kEnd && e + off < cE;
          uint32_t p = go ? e + off : kAway, kk = 0;
          uint32_t nn = 0, nruns = 0;  // notes; runs of empty blocks
          const uint32_t chunk = min((uint32_t)lane, NB - 1);
          uint16_t* const nt = s_note + chunk * (NOTES >> lg);
          uint16_t* const spare = s_note + NOTES + lane;  // a store here instead of a branch around one
          uint32_t over = kDead;  // how far past the chunk's end its chain crosses it
          do {
            uint32_t pp[5], b;
            pp[0] = p;
#pragma unroll
            for (int u = 0; u < 4; u++) pp[u + 1] = ch.next(pp[u], b);
            const bool room = nn + 4 <= NOTES >> lg;
            uint32_t n = 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const bool in = pp[u] < cE && pp[u + 1] < kAway;  // a block of the chunk with a valid header
              *(in && room ? nt + nn + u : spare) = (uint16_t)pp[u];
              n += in ? 1u : 0u;
              over = min(over, pp[u + 1] - cE);
            }
            kk += n;
            nn += room ? n : NOTES;  // too many: past the limit from here on
            p = pp[4];
            if (p - pp[0] == 4 * Chain<LPB, FM2>::kEmpty && p < cE) {  // a run of empty blocks is taken at once
              const uint32_t first = p, k0 = kk;
              ch.zeros(p, cE, kk);
              over = min(over, p - cE);
              if (kk != k0) {
                if (nruns < RUNS >> lg) {
                  s_runs[chunk * (RUNS >> lg) + nruns] = nn << 16 | first;
                  s_len[chunk * (RUNS >> lg) + nruns] = (uint16_t)(kk - k0);
                }
                nruns++;
              }
            }
          } while (__any_sync(0xffffffffu, p < cE));
          if (need) {
            k = kk;
            x = go ? (over > MAXSZ ? kDead : reg(cE + over)) : e;
            noted = nn <= NOTES >> lg && nruns <= RUNS >> lg;
            s_notes[lane] = nn | nruns << 16;
          }
          // A lane's entry is its predecessor's exit; one that was not goes again.  Of
          // neighbours that were not only the first goes (the others' predecessors are
          // to change), and none goes by a walk that died: that is most often one to
          // be mended itself, and the lanes behind it, which had been right, went the
          // same way one after the other, each a walk (4 us) of its own: 64 us in one of
          // the 1060 super-chunks of a segment, which the next 800 waited for.
          const uint32_t px = __shfl_up_sync(0xffffffffu, x, 1);
          differ = __ballot_sync(0xffffffffu, lane > 0 && act && px != e && px != kDead);
          need = (differ & ~(differ << 1)) >> lane & 1;
          if (need) {
            e = px;
            repaired = true;
          }
        } while (differ);
        // behind a walk that died on the chain itself there are no blocks
        const uint32_t dead = __ballot_sync(0xffffffffu, act && x == kDead);
        if (__builtin_expect(dead && act && lane >= __ffs(dead), false)) {
          e = x = kDead;
          k = 0;
          noted = true;
          s_notes[lane] = 0;
        }
        // exit, count and each lane's first block
        const uint32_t nact = __popc(__ballot_sync(0xffffffffu, act));
        xl = __shfl_sync(0xffffffffu, x, nact - 1);
        const uint32_t incl = warp_incl_scan(k, lane);
        K = __shfl_sync(0xffffffffu, incl, 31);
        const bool all_noted = __all_sync(0xffffffffu, noted);
        noted = all_noted && K <= KCAP;
        wi0 = incl - k;
        wn = incl;
        wp0 = e + off;  // e is a position where k > 0
        wi = wi0;
        wp = wp0;
        if (FM2 && known && !j0) {  // nothing else is needed: the tiles after this one wait for it
          if (lane == 0)
            publish(a.status + 2ull * s_t.rec, epoch, kFlagInclusive, cnt0 + K, 0u, h0, xl, scS, scE);
        }
        if (lane < (int)NB) s_c0[lane] = wi0;
        if (lane == 0) {
          s_c0[NB] = K;
          s_k = K;
          s_h0 = h0;
          s_noted = noted;
          s_many = all_noted && K > KCAP;
        }
        if (__builtin_expect(!all_noted, false)) list(0);
      }
      __syncthreads();
      if (s_noted) {  // gather the lanes' notes
        const uint32_t i = tid * (1u << lg) / kFlowThreads, TPC = kFlowThreads >> lg;  // threads per chunk
        const uint32_t c0 = s_c0[i], n = s_c0[i + 1] - c0;
        const uint16_t* const nt = s_note + i * (NOTES >> lg);
        const uint32_t r0 = i * (RUNS >> lg);
        const uint32_t nn = n ? s_notes[i] & 0xFFFFu : 0u, nruns = n ? s_notes[i] >> 16 : 0u;
        if (nruns == 0) {
          for (uint32_t t = tid & (TPC - 1); t < nn; t += TPC) s_pos[c0 + t] = nt[t];
        } else {  // between its runs of empty blocks
          uint32_t t0 = 0, at = c0;
          for (uint32_t g = 0; g <= nruns; g++) {
            const uint32_t run = g < nruns ? s_runs[r0 + g] : nn << 16, len = g < nruns ? s_len[r0 + g] : 0u;
            const uint32_t t1 = run >> 16;
            for (uint32_t t = t0 + (tid & (TPC - 1)); t < t1; t += TPC) s_pos[at + t - t0] = nt[t];
            at += t1 - t0;
            for (uint32_t t = tid & (TPC - 1); t < len; t += TPC) s_pos[at + t] = (uint16_t)((run & 0xFFFFu) + t * Chain<LPB, FM2>::kEmpty);
            at += len;
            t0 = t1;
          }
        }
        __syncthreads();
      }
      K = s_k;
      sum = 0;
      for (uint32_t kb = 0; kb < K && !FM2; kb += KCAP) {
        if (__builtin_expect(kb || s_many, false)) {
          __syncthreads();
          if (s_many) {
            gather_window(s_pos, s_note, s_notes, s_runs, s_len, s_c0, NOTES >> lg, RUNS >> lg, lg, kb, KCAP, Chain<LPB, FM2>::kEmpty);
          } else if (warp == 0) {
            list(kb);
          }
          __syncthreads();
        }
        sum += sums(min(KCAP, K - kb));
      }
      const uint32_t rec = s_t.rec;  // the records of a segment follow one another
      uint64_t* const st = a.status + 2ull * rec;
      if (known) {
        if (j0) base = s_t.seed;
        if (tid == 0 && (!FM2 || j0)) publish(st, epoch, kFlagInclusive, cnt0 + K, base + sum, h0, xl, scS, scE);
        break;
      }
      if (tid == 0) publish(st, epoch, kind, K, sum, h0, xl, scS, scE);
      h0 = s_h0;
      // Lane l of warp 0 reads the record at distance 1 + l; where none of those 32
      // is inclusive (a stream of one segment has all the CTAs in flight behind one
      // another) the four warps go on with 128 records a trip.  (Four windows from
      // the start: 255 us instead of 232 on 134 M values in 16 segments.)
      // A window that is not ready is read again; a broken chain of (entry, exit)
      // pairs (an older tile will correct itself) starts the look-back over.  A
      // tile whose entry is not its neighbour's exit walks again at once, from that
      // exit (if it is one: no tile gives up an entry for a walk that went wrong),
      // and publishes a second aggregate, so that the wrong entries of a segment
      // are mended side by side and not each after the prefixes of the one before
      // (2 M values of one segment whose entries are often wrong: 123 -> 85 us;
      // 134 M values in 16 segments 233 -> 225).  When that was not the true entry either,
      // the next walk waits until the whole chain is known.
      const int64_t first = (int64_t)rec - s_t.j;
      const uint32_t sc = s_t.sc;
      const bool may_second = (s_epoch & 0xFFFFF) != 0;  // a zeroed word must not read as a second claim
      uint32_t spins = 0, pred_x = kDead, need_x = h0;
      bool self_ok = true;
      int verdict = 0;  // 1 done, 2 entry unlike the neighbour's exit, 3 own entry wrong
      int64_t at = (int64_t)rec - 1;
      cnt0 = 0;
      base = 0;
      while (verdict == 0) {
        const int span = at == (int64_t)rec - 1 ? 1 : kFlowWarps;
        const int64_t mine = at - 32 * warp, idx = mine - lane;
        if (warp < span && mine >= first) {
          const bool inr = idx >= first;
          ulonglong2 w = make_ulonglong2(0, 0);
          uint64_t f = 0;
          uint32_t bi = 0;
          bool wait;
          while (true) {
            if (inr) w = ld_record(a.status + 2 * idx);
            f = status_flag(w.x);
            const bool ready = !inr || (w.x >> 42 == w.y >> 42 && status_epoch(w.x) == (s_epoch & 0xFFFFF) &&
                                        (f == kFlagAggregate || f == kFlagInclusive || f == kFlagSecond && may_second));
            bi = __ballot_sync(0xffffffffu, inr && ready && f == kFlagInclusive);
            wait = __any_sync(0xffffffffu, inr && !ready && lane < (bi ? __ffs(bi) : 32));
            if (!wait || ++spins > kSpinLimit || ((spins & 63) == 0 && launch_gave_up(a.err))) break;
            __nanosleep(100);
          }
          const bool incl = inr && f == kFlagInclusive;  // (only looked at where the record is ready)
          const int jstar = bi ? __ffs(bi) - 1 : 32;     // nearest inclusive of the window
          const bool rel = inr && lane <= jstar;
          const uint64_t vx = status_value(w.x), vy = status_value(w.y);
          const uint32_t tS = (uint32_t)(idx - first) * sc, tE = tS + min(sc, rlen - tS);
          const uint32_t xr = (uint32_t)(vx & 1023u) | (uint32_t)(vy & 1023u) << 10;
          const uint32_t tx = xr == kXDead ? kDead : xr == kXEnd ? kEnd : tE + xr;
          const uint32_t hr = (uint32_t)(vx >> 26) & 0xFFFFu;
          const uint32_t th = hr == kHDead ? kDead : hr == kHEnd ? kEnd : tS + hr;
          const uint32_t cnt = incl ? (uint32_t)(vx >> 10) : (uint32_t)(vx >> 10) & 0xFFFFu;
          // the entry of a lane's tile must be the exit of the next older one
          const uint32_t ox = __shfl_down_sync(0xffffffffu, tx, 1);
          const bool bad = __any_sync(0xffffffffu, rel && lane < jstar && lane < 31 && idx - 1 >= first && th != ox);
          // counts of up to 2^32 - 1 in all: a segment's region is below 4 GiB
          const uint32_t c = __reduce_add_sync(0xffffffffu, rel ? cnt : 0u);
          const uint32_t s = __reduce_add_sync(0xffffffffu, rel ? (uint32_t)(vy >> 10) : 0u);
          if (lane == 0) {
            s_win[warp].state = wait ? 1u : bad ? 2u : jstar < 32 ? 3u : 0u;
            s_win[warp].cnt = c;
            s_win[warp].sum = s;
            s_win[warp].exit = tx;
          }
          if (lane == 31) s_win[warp].entry = th;
        }
        __syncthreads();
        // every thread takes the windows together, nearest first
        bool over = false;
        for (int v = 0; v < span && verdict == 0; v++) {
          const FlowWindow& win = s_win[v];
          if (win.state == 1) {  // not ready for too long
            if (tid == 0) atomicOr(a.err, kErrLookbackTimeout);
            verdict = 1;
            break;
          }
          if (at == (int64_t)rec - 1) {
            self_ok = win.exit == h0;
            pred_x = win.exit;
            if (!self_ok && kind == kFlagAggregate && may_second && pred_x < kEnd) {
              verdict = 2;
              break;
            }
          } else if (win.exit != need_x) {
            over = true;
          }
          if (win.state == 2 || over) {
            over = true;
            break;
          }
          cnt0 += win.cnt;
          base += win.sum;
          need_x = win.entry;
          at -= 32;
          if (win.state == 3 || at < first) verdict = self_ok ? 1 : 3;
        }
        __syncthreads();  // the windows are read before they are written again
        if (verdict == 0 && over) {
          const bool give_up = ++spins > kSpinLimit || ((spins & 63) == 0 && launch_gave_up(a.err));
          if (__syncthreads_or(give_up)) {
            if (tid == 0) atomicOr(a.err, kErrLookbackTimeout);
            verdict = 1;
          } else {
            at = (int64_t)rec - 1;
            need_x = h0;
            cnt0 = 0;
            base = 0;
            __nanosleep(200);
          }
        }
      }
      if (verdict >= 2) {
        known = verdict == 3;
        kind = kFlagSecond;
        if (tid == 0) {  // unready until the corrected record is out
          st_relaxed_u64(st, make_status(epoch, 3, 0));
          st_relaxed_u64(st + 1, make_status(epoch, 3, 0));
        }
        h0 = pred_x;
        repaired = true;
        continue;
      }
      if (tid == 0) publish(st, epoch, kFlagInclusive, cnt0 + K, base + sum, h0, xl, scS, scE);
      break;
    }
    __syncthreads();  // the groups' prefixes are in place
    if (warp == 0) {
      if (__any_sync(0xffffffffu, repaired) && lane == 0) atomicAdd(&a.counters[0], 1u);
      if (lane == 0 && s_t.last) {  // the last super-chunk of a segment checks the block total
        const uint64_t all = cnt0 + K;
        if (all < s_t.nb || (s_t.strict && all != s_t.nb)) atomicOr(s_t.err, kErrBlockCount);
      }
    }
    // ---- decode ----
    const uint64_t g0 = cnt0, nb = s_t.nb;  // the blocks before the super-chunk
    const uint32_t kmax = g0 >= nb ? 0u : (uint32_t)min((uint64_t)K, nb - g0);
    Put<OUT> put(s_t.eb, s_t.ebd);
    using E = typename Elem<OUT>::T;
    E* const y = static_cast<E*>(s_t.y) + s_t.lo;  // block g's values start at y + g*L (fastmode1: with the value before it)
    uint32_t qpass = base;
    bool corrupt = false;
    for (uint32_t kb = 0; kb < kmax; kb += KCAP) {
      const uint32_t kn = min(KCAP, kmax - kb);
      if (__builtin_expect(K > KCAP, false)) {  // more blocks than the list holds: list them again
        __syncthreads();
        if (s_many) {
          gather_window(s_pos, s_note, s_notes, s_runs, s_len, s_c0, NOTES >> lg, RUNS >> lg, lg, kb, KCAP, Chain<LPB, FM2>::kEmpty);
        } else if (warp == 0) {
          if (kb == 0) {
            wi = wi0;
            wp = wp0;
          }
          list(kb);
        }
        __syncthreads();
        const uint32_t run = sums(min(KCAP, K - kb));
        if (tid == 0) s_sum = run;
        __syncthreads();
      }
      const uint32_t ng = (kn + BPR - 1) / BPR;                           // groups listed
      const bool tail = g0 + kb + (uint64_t)ng * BPR >= nb;               // the last one holds the segment's last block
      const uint32_t nfast = tail ? ng - 1 : ng;
      // two neighbouring groups at a time: their chains of loads, votes and shuffles overlap
      for (uint32_t r = 2 * warp; r < nfast; r += 2 * kFlowWarps) {
        uint32_t o[2], bc[2], seed[2], q[2][8];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const uint32_t ru = min(r + u, nfast - 1), blk = (r + u) * BPR + grp;
          const bool valid = r + u < nfast && blk < kn;
          o[u] = s_pos[valid ? blk : r * BPR];
          seed[u] = 0;
          if (FM2) {
            seed[u] = lds_le32(s_b, o[u]);
            o[u] += 4;
          } else {
            seed[u] = qpass + s_tot[ru];  // the value before the group
          }
          bc[u] = valid ? s_b[o[u]] : 0u;
        }
        const uint32_t top = __reduce_max_sync(0xffffffffu, max(bc[0], bc[1]));
        // q: the value before each of the lane's deltas
        auto groups = [&](auto planes) {
          constexpr int PL = decltype(planes)::value;
          const Deltas<LPB, FM2, PL> d[2] = {{s_b, o[0], bc[0], sub}, {s_b, o[1], bc[1], sub}};
          uint32_t incl[2] = {d[0].total, d[1].total};
          constexpr int SW = FM2 ? LPB : 32;  // lanes whose deltas add up: the block's, or the group's
#pragma unroll
          for (int s = 1; s < SW; s <<= 1) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
              const uint32_t v = __shfl_up_sync(0xffffffffu, incl[u], s, SW);
              if (lane % SW >= s) incl[u] += v;
            }
          }
#pragma unroll
          for (int u = 0; u < 2; u++) d[u].before(seed[u] + incl[u] - d[u].total, q[u]);
        };
        if (top == 0) {  // empty blocks
#pragma unroll
          for (int u = 0; u < 2; u++)
#pragma unroll
            for (int i = 0; i < 8; i++) q[u][i] = seed[u];
        } else if (top < 8) {
          groups(std::integral_constant<int, 0>{});
        } else if (top < 16) {
          groups(std::integral_constant<int, 1>{});
        } else if (top < 24) {
          groups(std::integral_constant<int, 2>{});
        } else {
          groups(std::integral_constant<int, 3>{});
        }
        const uint32_t blocks = min(min(2u, nfast - r) * BPR, kn - r * BPR);
        store_groups<OUT>(put, y + (g0 + kb + (uint64_t)r * BPR) * L, q, blocks * LPB, lane, s_tried[warp]);
      }
      if (tail && (ng - 1) % kFlowWarps == (uint32_t)warp) {
        const uint32_t r = ng - 1, blk = r * BPR + grp;
        const bool valid = blk < kn;
        uint32_t o = s_pos[valid ? blk : r * BPR];
        const uint64_t g = g0 + kb + r * BPR;  // the group's first block
        const uint32_t bq = FM2 ? 0u : qpass + s_tot[r];
        {
          // ---- the group that holds the segment's last block ----
          const uint64_t b0 = (g + grp) * L;  // element of y before (fastmode1) or at (fastmode2) the block's first
          const uint64_t len = s_t.hi - s_t.lo;
          const uint32_t m = valid ? (uint32_t)min((uint64_t)(FM2 ? L - 1 : L), len - 1 - b0) : 0u;  // packed values
          const uint32_t ml = m > 8u * sub ? min(8u, m - 8u * sub) : 0u;
          uint32_t d[8], run = 0, seed = 0, bc = 0;
          if (FM2) {
            if (valid) {
              if (rlen - (o - off) < 4) {
                corrupt = true;
              } else {
                seed = lds_le32(s_b, o);
              }
            }
            o += 4;
          }
          if (m) {
            bc = o - off < rlen ? s_b[o] : 255u;
            if (bc > 33 || block_bytes(m, bc) > rlen - (o - off)) {
              corrupt = true;
              bc = 0;
            }
          }
          unpack_any<LPB>(s_b, o, bc, m, ml, sub, d);
          uint32_t w[9];
#pragma unroll
          for (int i = 0; i < 8; i++) {
            w[i] = run;
            run += d[i];
          }
          w[8] = run;
          uint32_t q0;
          if (FM2) {
            uint32_t incl = run;
#pragma unroll
            for (int s = 1; s < LPB; s <<= 1) {
              const uint32_t v = __shfl_up_sync(0xffffffffu, incl, s, LPB);
              if (sub >= s) incl += v;
            }
            q0 = seed + incl - run;
          } else {
            q0 = bq + warp_incl_scan(run, lane) - run;
          }
          if (valid) {
            const uint32_t top = FM2 || g + grp + 1 == nb ? m : L - 1;  // fastmode1: the next block stores this one's last
#pragma unroll
            for (int i = 0; i < 9; i++)
              if ((i < 8 || sub == LPB - 1) && 8u * sub + i <= top) put.one(y, b0 + 8 * sub + i, q0 + w[i]);
          }
        }
      }
      if (K > KCAP) qpass += s_sum;
    }
    if (__any_sync(0xffffffffu, corrupt) && lane == 0) atomicOr(s_t.err, kErrCorrupt);
    if (OUT == kOutCodesAdd && __any_sync(0xffffffffu, put.wrap) && lane == 0) atomicOr(s_t.err, kErrQuantRange);
  }
}

template <int LPB, bool BATCH, bool FM2, int OUT>
cudaError_t launch_one(const DecArgs& a, cudaStream_t st) {
  auto k = decode_flow<LPB, BATCH, FM2, OUT>;
  const size_t smem = flow_smem<LPB, FM2>();
  // resident CTAs of this instance, cached per device as (device + 1) << 32 | CTAs
  static std::atomic<uint64_t> s_cache{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  uint64_t c = s_cache.load(std::memory_order_relaxed);
  if ((c >> 32) != (uint64_t)dev + 1) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int occ = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kFlowThreads, smem);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    c = ((uint64_t)dev + 1) << 32 | (uint32_t)((occ < 1 ? 1 : occ) * sms);
    s_cache.store(c, std::memory_order_relaxed);
  }
  const uint32_t cap = (uint32_t)c;
  const uint32_t grid = a.nlocate_ctas < cap ? a.nlocate_ctas : cap;
  if (grid == 0) return cudaSuccess;
  if (!BATCH) return launch_behind(k, grid, kFlowThreads, smem, st, a);
  k<<<grid, kFlowThreads, smem, st>>>(a);
  return cudaGetLastError();
}

template <bool FM2, int OUT>
cudaError_t launch_lpb(const DecArgs& a, cudaStream_t st) {
  switch (a.f.seg.L) {
    case 8: return launch_one<1, false, FM2, OUT>(a, st);
    case 16: return launch_one<2, false, FM2, OUT>(a, st);
    case 32: return launch_one<4, false, FM2, OUT>(a, st);
    case 64: return launch_one<8, false, FM2, OUT>(a, st);
    case 128: return launch_one<16, false, FM2, OUT>(a, st);
    case 256: return launch_one<32, false, FM2, OUT>(a, st);
    default: return cudaErrorInvalidValue;
  }
}

template <bool FM2>
cudaError_t launch_out(const DecArgs& a, cudaStream_t st) {
  switch (a.out_kind) {
    case kOutFloat: return launch_lpb<FM2, kOutFloat>(a, st);
    case kOutDouble: return launch_lpb<FM2, kOutDouble>(a, st);
    case kOutCodes: return launch_lpb<FM2, kOutCodes>(a, st);
    default: return launch_lpb<FM2, kOutCodesAdd>(a, st);
  }
}

}  // namespace

bool flow_supported(uint32_t L) { return L >= 8 && L <= 256 && (L & (L - 1)) == 0; }

uint32_t flow_chunk_bytes(uint32_t L) {
  switch (L) {
    case 64: return Shape<8>::C;
    case 128: return Shape<16>::C;
    case 256: return Shape<32>::C;
    default: return Shape<4>::C;
  }
}

cudaError_t launch_decode_flow(const DecArgs& a, cudaStream_t st) {
  return a.fm2 ? launch_out<true>(a, st) : launch_out<false>(a, st);
}

// Batched fastmode1 decode, blockSize 32.
cudaError_t launch_decode_flow_batch(const DecArgs& a, cudaStream_t st) {
  return launch_one<4, true, false, kOutFloat>(a, st);
}

// Sets the batched decoder's shared-memory limit and caches its grid without
// launching anything (no super-chunks), so that no later launch does that work.
cudaError_t prepare_decompress_batch() {
  DecArgs a;
  memset(&a, 0, sizeof a);
  return launch_decode_flow_batch(a, 0);
}

}  // namespace szp
