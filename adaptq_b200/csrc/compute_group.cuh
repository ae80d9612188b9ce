// Decode attention for grouped queries: several queries of one KV head in one pass over its
// cache (2-, 3- or 4-bit K and V at padded dimension 64 or 128; dense V).
//
// Replaces the same upstream code as compute_general.cuh and compute_stream.cuh -- the quantised
// branch of AttentionHead::compute (attention/attention.cpp:526-563, :606-633) with compute_avx2
// (:373-474) -- for the calls that upstream makes once per query (adaptq_mha_compute_batch).
// compute_stream.cuh reads the packed rows through score tables and buckets in shared memory,
// one lookup per packed byte AND query, so its time grows with the queries.  Here the packed
// rows are turned into operands of the tensor cores once and contracted with all queries:
//
//  * The arithmetic is in integers.  The centroids are four-decimal numbers: 10^4 * centroid is a
//    16-bit integer = two signed bytes ("planes").  A rotated query is a 31-bit fixed-point number
//    relative to its largest coordinate = four signed bytes ("digits"), a token's weight a 31-bit
//    number relative to its chunk's total = four unsigned ones.  mma.sync m16n8k32 on bytes with
//    32-bit sums contracts 16 rows with the digits of two queries: a column collects one place
//    256^k, to which the high plane brings one digit and the low plane the next, so both planes
//    share a sum; the places are put together in floats (K) or 64-bit integers (V).
//  * K scores: rows = tokens, k = coordinates.  V: rows = coordinates, k = tokens.
//  * 4-bit codes become plane bytes through a table in shared memory, one lookup per packed byte
//    (two coordinates, both planes), each lane in its own bank; 2- and 3-bit codes through byte
//    permutes with the code as selector.  2-bit values need no table at all: their codebook is
//    linear in the two bits, so the bits themselves are the planes.
//  * A block runs two independent groups (eight consumer warps and a producer warp each): one
//    streams while the other is at its softmax.  A group walks a contiguous run of 64-token
//    units of the call's (head, query group) list, cut anywhere, so all groups finish together;
//    what a group holds of one head is a segment, walked in chunks of at most CHUNK tokens:
//    K rows (scores to shared memory), exact softmax of the chunk, V rows, then a
//    rescale-and-add onto the segment's float accumulator.  A head that one group holds alone is
//    finished there; otherwise the group that brings a query's arrival count to the number of
//    segments merges their partials (nobody waits for anybody).
//
// What bounds it (512 heads x 4096 tokens, K4/V2, dim 128, four queries: 110 us, 27 warp
// instructions per token): the 16 warps that 64 accumulators and 32 operand registers a thread leave
// room for keep the issue slots half busy; integer pipe 41 %, shared-memory wavefronts 43 %, tensor
// pipe 30 %.  Of a warp's time the K stream takes 35 %, the V stream 24 %, softmax and weights 17 %,
// the ends of segments 18 %.
#pragma once
#include "common.cuh"
#include "compute_stream.cuh"

namespace aq {

constexpr int GQ_WARPS = 8;                       // consumer warps of a group
constexpr int GQ_GROUP_THREADS = GQ_WARPS * 32;
constexpr int GQ_GROUPS = 2;                      // independent groups per block
// 16 consumer warps, then a warpgroup whose first two warps are the groups' producers.  The block is
// launched with 96 registers a thread (five warps share a quarter SM's 16,384); the producers'
// warpgroup gives its share back: 512 * 112 + 128 * 32 = the launch's 61,440.
constexpr int GQ_THREADS = GQ_GROUPS * GQ_GROUP_THREADS + 128;
constexpr int GQ_REGS_CONSUMER = 112, GQ_REGS_PRODUCER = 32;
static_assert(GQ_GROUPS * GQ_GROUP_THREADS * GQ_REGS_CONSUMER + 128 * GQ_REGS_PRODUCER <= GQ_THREADS * 96, "register split");
constexpr int GQ_UNIT = 64;                       // tokens per unit of the work split: copies stay 16-byte aligned
constexpr int GQ_STAGE = 8192;                    // bytes of packed rows per ring stage
constexpr int GQ_TABLE = 65536;                   // 256 entries x 256 bytes (the first 32 words hold the entry, one per lane)
constexpr size_t GQ_SMEM_MAX = 232448;

struct GroupLaunch {
  CacheView c;
  const float *q;  // [heads_in_call][nq][dim]
  float *out;      // [heads_in_call][nq][dim]
  float *partial;  // [runs][2][per_group][2+P]: pieces of cut heads, 0 where the piece starts its group's run, else 1
  int *counters;   // [heads_in_call*nq] arrival counts, zero before and after every launch
  int head0, heads_in_call, nq;
  int groups_per_head, per_group; // query groups of a head and queries per group (the last may have fewer)
  int n;           // live tokens
  int units;       // units per item, and the tokens of one unit
  int unit_tokens;
  int *status;
};

// 10^4 * centroid = 256 * (high plane) + (low plane), both signed bytes.
template <int BITS> __host__ __device__ constexpr int gq_magnitude(int i) {
  if (BITS == 2) return i == 0 ? 4528 : 15104;
  if (BITS == 3) return i == 0 ? 2451 : i == 1 ? 7560 : i == 2 ? 13439 : 21529;
  return i == 0 ? 1258 : i == 1 ? 3795 : i == 2 ? 6402 : i == 3 ? 9138 : i == 4 ? 12016 : i == 5 ? 15105 : i == 6 ? 18944 : 24008;
}
template <int BITS> __host__ __device__ constexpr int gq_value(int code) {
  return code >= (1 << (BITS - 1)) ? gq_magnitude<BITS>(code - (1 << (BITS - 1))) : -gq_magnitude<BITS>((1 << (BITS - 1)) - 1 - code);
}
template <int BITS> __host__ __device__ constexpr uint32_t gq_plane(int code, int high) { // as a byte
  const int shifted = gq_value<BITS>(code) + 128 + 65536; // positive, so that the division rounds down
  return (uint32_t)(high ? shifted / 256 - 256 : shifted % 256 - 128) & 255u;
}
// plane bytes of codes first..first+3
template <int BITS> __host__ __device__ constexpr uint32_t gq_plane_word(int first, int high) {
  uint32_t w = 0;
  for (int k = 0; k < 4; ++k) w |= gq_plane<BITS>(first + k, high) << (8 * k);
  return w;
}

#define GQ_MMA(name, ta, tb)                                                                                              \
  __device__ __forceinline__ void name(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) { \
    asm("mma.sync.aligned.m16n8k32.row.col.s32." ta "." tb ".s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"    \
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])                                                                   \
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));                                                           \
  }
GQ_MMA(mma_s8s8, "s8", "s8")
GQ_MMA(mma_s8u8, "s8", "u8")
GQ_MMA(mma_u8u8, "u8", "u8")
#undef GQ_MMA
// Byte permute with a computed selector whose nibbles are known to be below 8.
__device__ __forceinline__ uint32_t prmt_sel(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// Eight 3-bit codes (bits 0..23, first code on top; the top byte is ignored) -> eight nibbles,
// nibble n = code 7-n.
__device__ __forceinline__ uint32_t spread3(uint32_t v24) {
  uint32_t x = (v24 & 0x00000FFFu) | ((v24 << 4) & 0x0FFF0000u);
  x = (x & 0x003F003Fu) | ((x << 2) & 0x3F003F00u);
  return (x & 0x07070707u) | ((x << 1) & 0x70707070u);
}

// Operand registers of the K stream.  A lane (tig = lane & 3) contributes a quarter of a row, P/4
// coordinates, as P/8 registers of four bytes.  4 bits: register r = one packed byte, {high, low}
// planes of its two coordinates.  2 and 3 bits: register 2i = the high planes of four coordinates,
// 2i + 1 = the low planes of the same.  k_coord: the coordinate that byte b of register r belongs to.
template <int KB, int P> __device__ __forceinline__ int k_coord(int tig, int r, int b) {
  if (KB == 4) return tig * (P / 4) + 2 * r + (b >> 1);
  const int i = r >> 1;
  if (KB == 3) return tig * (P / 4) + (i >> 1) * 8 + ((i & 1) ? 3 - b : 7 - b);
  // 2 bits: a word of 16 codes gives four registers: odd positions of bytes 0,1 and 2,3, then the even ones
  return tig * (P / 4) + (i >> 2) * 16 + (i & 1) * 8 + (b >> 1) * 4 + ((b & 1) ? 0 : 2) + ((i & 2) ? 0 : 1);
}

// Raw words of one row that this lane contributes (its P/4 coordinates).
template <int KB, int P> struct KLane {
  static constexpr int WORDS = KB == 3 ? (P == 128 ? 3 : 2) : P / 4 * KB / 32;
};
template <int KB, int P>
__device__ __forceinline__ void load_k_lane(const uint8_t *row, int tig, uint32_t (&w)[KLane<KB, P>::WORDS]) {
  constexpr int W = KLane<KB, P>::WORDS;
  if constexpr (W == 4) {
    const uint4 v = *reinterpret_cast<const uint4 *>(row + tig * 16);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else if constexpr (KB == 3 && P == 64) { // six bytes at 6*tig: two aligned words around them
    const uint32_t *r = reinterpret_cast<const uint32_t *>(row) + ((6 * tig) >> 2);
    w[0] = r[0]; w[1] = r[1];
  } else if constexpr (W == 3) {
    const uint32_t *r = reinterpret_cast<const uint32_t *>(row) + 3 * tig;
    w[0] = r[0]; w[1] = r[1]; w[2] = r[2];
  } else if constexpr (W == 2) {
    const uint2 v = *reinterpret_cast<const uint2 *>(row + tig * 8);
    w[0] = v.x; w[1] = v.y;
  } else {
    w[0] = *reinterpret_cast<const uint32_t *>(row + tig * 4);
  }
}

template <int KB, int P>
__device__ __forceinline__ void expand_k(const uint32_t (&w)[KLane<KB, P>::WORDS], int tig, uint32_t lane_table, uint32_t (&ar)[P / 8]) {
  if constexpr (KB == 4) { // table address = {lane column, code byte, table base}: one permute, one lookup per packed byte
#pragma unroll
    for (int m = 0; m < P / 32; ++m) {
#pragma unroll
      for (int k = 0; k < 4; ++k) ar[4 * m + k] = lds_u32(__byte_perm(w[m], lane_table, 0x7604 | (k << 4)));
    }
  } else if constexpr (KB == 3) {
    constexpr uint32_t H0 = gq_plane_word<3>(0, 1), H1 = gq_plane_word<3>(4, 1), L0 = gq_plane_word<3>(0, 0), L1 = gq_plane_word<3>(4, 0);
    uint32_t g[P / 32]; // eight codes each in bits 0..23, first byte on top
    if constexpr (P == 128) {
      g[0] = __byte_perm(w[0], 0u, 0x4012);
      g[1] = __byte_perm(w[0], w[1], 0x0345);
      g[2] = __byte_perm(w[1], w[2], 0x0234);
      g[3] = __byte_perm(w[2], 0u, 0x4123);
    } else {
      const uint32_t s0 = (tig & 1) ? 0x0234u : 0x0012u, s1 = (tig & 1) ? 0x0567u : 0x0345u;
      g[0] = prmt_sel(w[0], w[1], s0);
      g[1] = prmt_sel(w[0], w[1], s1);
    }
#pragma unroll
    for (int m = 0; m < P / 32; ++m) {
      const uint32_t x = spread3(g[m]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t s = h ? x >> 16 : x;
        ar[2 * (2 * m + h)] = prmt_sel(H0, H1, s);
        ar[2 * (2 * m + h) + 1] = prmt_sel(L0, L1, s);
      }
    }
  } else {
    constexpr uint32_t H0 = gq_plane_word<2>(0, 1), L0 = gq_plane_word<2>(0, 0);
#pragma unroll
    for (int m = 0; m < P / 64; ++m) {
      const uint32_t a = w[m] & 0x33333333u, b = (w[m] >> 2) & 0x33333333u;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t x = (r & 2) ? b : a, s = (r & 1) ? x >> 16 : x;
        ar[2 * (4 * m + r)] = prmt_sel(H0, 0u, s);
        ar[2 * (4 * m + r) + 1] = prmt_sel(L0, 0u, s);
      }
    }
  }
}

// V stream: a lane owns unit u (eight consecutive coordinates = VB bytes) of four tokens at a time.
template <int VB> struct VWords { static constexpr int N = VB == 3 ? 2 : 1; };
template <int VB, int P> __device__ __forceinline__ void load_v_unit(const uint8_t *row, int u, uint32_t (&w)[VWords<VB>::N]) {
  if constexpr (VB == 4) w[0] = reinterpret_cast<const uint32_t *>(row)[u];
  else if constexpr (VB == 2) w[0] = reinterpret_cast<const uint32_t *>(row)[u >> 1];
  else {
    const int i = (3 * u) >> 2; // three bytes at 3*u: the word they start in and the next (within the row)
    w[0] = reinterpret_cast<const uint32_t *>(row)[i];
    w[1] = reinterpret_cast<const uint32_t *>(row)[min(i + 1, P * 3 / 32 - 1)];
  }
}
// First step, once per four tokens: the words that plane_pair() works on.
template <int VB> __device__ __forceinline__ void gather_v(const uint32_t (&w)[4][VWords<VB>::N], uint32_t usel, uint32_t (&x)[4]) {
  if constexpr (VB == 2) { // usel picks the unit's two bytes of both tokens: {t0.b0, t1.b0, t0.b1, t1.b1}
    const uint32_t t01 = prmt_sel(w[0][0], w[1][0], usel), t23 = prmt_sel(w[2][0], w[3][0], usel);
    x[0] = __byte_perm(t01, t23, 0x5410);
    x[1] = __byte_perm(t01, t23, 0x7632);
  } else if constexpr (VB == 4) {
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = w[t][0];
  } else { // nibbles of two tokens side by side: even nibbles of tokens 0/1, 2/3, odd nibbles of 0/1, 2/3
    uint32_t y[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) y[t] = spread3(prmt_sel(w[t][0], w[t][1], usel));
    x[0] = (y[0] & 0x0F0F0F0Fu) | ((y[1] << 4) & 0xF0F0F0F0u);
    x[1] = (y[2] & 0x0F0F0F0Fu) | ((y[3] << 4) & 0xF0F0F0F0u);
    x[2] = ((y[0] >> 4) & 0x0F0F0F0Fu) | (y[1] & 0xF0F0F0F0u);
    x[3] = ((y[2] >> 4) & 0x0F0F0F0Fu) | (y[3] & 0xF0F0F0F0u);
  }
}
// Coordinates 2*i and 2*i + 1 of the unit for the four tokens, two registers each: u[k], v[k].
// 2 and 3 bits: u = one plane of the four tokens, v = the other; 4 bits: u = {high, low} planes of
// tokens 0 and 1, v of tokens 2 and 3.
template <int VB>
__device__ __forceinline__ void plane_pair(const uint32_t (&x)[4], int i, uint32_t lane_table, uint32_t (&u)[2], uint32_t (&v)[2]) {
  if constexpr (VB == 2) { // the bits stay where they are: the sums carry a factor 2^position
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int s = 2 * i + k;
      u[k] = x[s >> 2] & (0x80808080u >> (2 * (s & 3)));
      v[k] = x[s >> 2] & (0x40404040u >> (2 * (s & 3)));
    }
  } else if constexpr (VB == 4) {
    uint32_t e[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) e[t] = lds_u32(__byte_perm(x[t], lane_table, 0x7604 | (i << 4)));
    u[0] = __byte_perm(e[0], e[1], 0x5410);
    u[1] = __byte_perm(e[0], e[1], 0x7632);
    v[0] = __byte_perm(e[2], e[3], 0x5410);
    v[1] = __byte_perm(e[2], e[3], 0x7632);
  } else {
    constexpr uint32_t H0 = gq_plane_word<3>(0, 1), H1 = gq_plane_word<3>(4, 1), L0 = gq_plane_word<3>(0, 0), L1 = gq_plane_word<3>(4, 0);
#pragma unroll
    for (int k = 0; k < 2; ++k) { // nibble 7 - s holds coordinate s = 2*i + k: byte 3 - i, the odd one first
      const int by = 3 - i;
      const uint32_t sel = k == 0 ? __byte_perm(x[2], x[3], by | ((4 + by) << 4)) : __byte_perm(x[0], x[1], by | ((4 + by) << 4));
      u[k] = prmt_sel(H0, H1, sel);
      v[k] = prmt_sel(L0, L1, sel);
    }
  }
}

// Shared-memory plan of one instantiation.  With a 4-bit side the lookup table sits on a 64 KB
// boundary (a byte permute then forms an address) with the integer sums in the unused halves of its
// entries; group 0's ring lies in front of it, everything else behind it.
template <int KB, int VB, int P, int NT> struct GroupPlan {
  static constexpr int NQ = 2 * NT;
  static constexpr int CHUNK = NT == 1 ? 2048 : 1536;
  static constexpr bool TABLE = KB == 4 || VB == 4;
  static constexpr int KROW = P * KB / 8, VROW = P * VB / 8;
  // tokens per stage; 3-bit rows fill three quarters of one
  static constexpr int TKN = KB == 3 ? GQ_STAGE * 3 / 4 / KROW : GQ_STAGE / KROW;
  static constexpr int TVN = VB == 3 ? GQ_STAGE * 3 / 4 / VROW : GQ_STAGE / VROW;
  static constexpr int SCORE_PITCH = CHUNK + 16;
  static constexpr int W_PITCH = CHUNK / 4 + 8; // words per (query, digit) plane of the weights
  static constexpr int SCORE_BYTES = NQ * (CHUNK + 32) * 4;
  static constexpr int PLANES = VB == 2 ? 2 : 1; // sums per (coordinate, column)
  static constexpr int SUM_ROWS = (P / 8) * 8 * PLANES * NT * 2 / 8; // rows of 32 words
  static constexpr int SUM_PITCH = TABLE ? 64 : 32;
  static constexpr int BQ_ROWS = NT * P / 8;
  static constexpr int MISC_BYTES = NQ * P * 4 + 1024 + BQ_ROWS * 128;
  static constexpr int STAGE_BYTES = GQ_STAGE + TKN * 4;
  static constexpr int STAGES = TABLE ? 4 : 6;
  static constexpr int RING = STAGES * STAGE_BYTES;
  static constexpr int GROUP_BYTES = RING + SCORE_BYTES + SUM_ROWS * 128 + MISC_BYTES; // without a table
  // in front of the table 63 KB are free (dynamic shared memory starts at 1 KB)
  static constexpr int BEHIND = 2 * (SCORE_BYTES + MISC_BYTES) + RING;
  static_assert(SCORE_BYTES % 128 == 0 && MISC_BYTES % 128 == 0 && STAGE_BYTES % 128 == 0, "alignment");
  static_assert(!TABLE || (RING <= 64512 && 2 * SUM_ROWS <= 256 && 64512 + GQ_TABLE + BEHIND <= (int)GQ_SMEM_MAX), "shared memory");
  static_assert(CHUNK % 64 == 0 && CHUNK * 4 <= STAGE_BYTES, "chunks keep the copies aligned; a chunk's V scales fit one stage");
  static_assert(CHUNK % (128 * (GQ_WARPS / NQ)) == 0, "whole quads per softmax thread");
  static constexpr size_t SMEM = TABLE ? GQ_SMEM_MAX : (size_t)GQ_GROUPS * GROUP_BYTES;
};

template <int KB, int VB, int P, int NT>
__global__ void __launch_bounds__(GQ_THREADS, 1) compute_group_kernel(const GroupLaunch a) {
  using PL = GroupPlan<KB, VB, P, NT>;
  constexpr int NQ = PL::NQ, CHUNK = PL::CHUNK, EPL = P / 32, KR = P / 8;
  extern __shared__ __align__(1024) unsigned char smem_group[];
  const int tid = threadIdx.x, lane = tid & 31, warp_all = tid >> 5;
  // warps 0..7 group 0, 8..15 group 1, 16 and 17 their producers (18 and 19 only complete the warpgroup)
  const bool producer = warp_all >= GQ_GROUPS * GQ_WARPS;
  const int grp = producer ? (warp_all - GQ_GROUPS * GQ_WARPS) % GQ_GROUPS : warp_all / GQ_WARPS;
  const int warp = warp_all % GQ_WARPS, gtid = tid % GQ_GROUP_THREADS;

  // ---- shared memory ----------------------------------------------------------------------------------
  uint32_t table_addr = 0, room = 0;
  bool layout_ok = true;
  if constexpr (PL::TABLE) {
    const uint32_t base = smem_u32(smem_group);
    table_addr = (base + 65535u) & ~65535u;
    room = table_addr - base;
    layout_ok = room >= (uint32_t)PL::RING && room + GQ_TABLE + PL::BEHIND <= (uint32_t)GQ_SMEM_MAX;
  }
  unsigned char *const behind = smem_group + room + GQ_TABLE; // scores and small variables of both groups, ring of group 1
  auto misc_of = [&](int g) -> unsigned char * {
    if (PL::TABLE) return behind + 2 * PL::SCORE_BYTES + (size_t)g * PL::MISC_BYTES;
    return smem_group + (size_t)(g + 1) * PL::GROUP_BYTES - PL::MISC_BYTES;
  };
  unsigned char *ring = PL::TABLE ? (grp == 0 ? smem_group : behind + PL::BEHIND - PL::RING) : smem_group + (size_t)grp * PL::GROUP_BYTES;
  float *sc = reinterpret_cast<float *>(PL::TABLE ? behind + (size_t)grp * PL::SCORE_BYTES : ring + PL::RING);
  uint32_t *wd = reinterpret_cast<uint32_t *>(sc); // the weights' digits take the scores' place
  uint32_t *sums = PL::TABLE ? reinterpret_cast<uint32_t *>(smem_group + room) + (size_t)grp * (PL::SUM_ROWS * PL::SUM_PITCH) + 32
                             : reinterpret_cast<uint32_t *>(ring + PL::RING + PL::SCORE_BYTES);
  int *qd = reinterpret_cast<int *>(misc_of(grp));          // [NQ][P] fixed-point rotated queries
  float *accb = reinterpret_cast<float *>(qd);              // row w is later warp w's finished accumulator
  uint32_t *bqs = reinterpret_cast<uint32_t *>(qd + NQ * P); // [BQ_ROWS][32] B operands of the K stream
  float *red = reinterpret_cast<float *>(bqs + PL::BQ_ROWS * 32); // [NQ][8] maxima | [8] sums | [8] weighted sums
  float *red_l = red + NQ * 8, *red_w = red_l + 8;
  uint32_t *wtot = reinterpret_cast<uint32_t *>(red_w + 8); // [8] integer totals of the weights
  float *qscale = reinterpret_cast<float *>(wtot + 8);      // [NQ]
  float *s_alpha = qscale + NQ, *s_scale = s_alpha + NQ, *s_m = s_scale + NQ, *s_l = s_m + NQ; // [NQ] each
  // a ring's barriers, and in group 0's part the failure flag, in the last 512 bytes
  auto bars_of = [&](int g) { return reinterpret_cast<uint64_t *>(misc_of(g) + PL::MISC_BYTES - 512); };
  uint64_t *full = bars_of(grp), *empty = full + PL::STAGES;
  volatile int *fail = reinterpret_cast<volatile int *>(bars_of(0) + 32);
  auto stage_ptr = [&](int s) { return ring + (size_t)s * PL::STAGE_BYTES; };

  if (!layout_ok) { // the same for every thread of the block: nothing is written
    if (tid == 0) atomicExch(a.status, 2);
    return;
  }
  if (tid == 0) {
    for (int g = 0; g < GQ_GROUPS; ++g)
      for (int s = 0; s < PL::STAGES; ++s) {
        mbar_init(bars_of(g) + s, 1);
        mbar_init(bars_of(g) + PL::STAGES + s, GQ_WARPS / 2);
      }
    *fail = 0;
    fence_barrier_init();
  }
  if constexpr (PL::TABLE) { // entry of a byte: {high, low} planes of its two codes, a copy for each lane
    uint32_t *t = reinterpret_cast<uint32_t *>(smem_group + room);
    for (int v = warp_all; v < 256; v += GQ_THREADS / 32) {
      uint32_t e = 0;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int x = __float2int_rn(c_cb[2][k ? v & 15 : v >> 4] * 10000.f), high = (x + 128 + 65536) / 256 - 256;
        e |= (((uint32_t)high & 255u) | (((uint32_t)(x - 256 * high) & 255u) << 8)) << (16 * k);
      }
      t[v * 64 + lane] = e;
    }
  }
  if (!producer)
    for (int i = warp; i < PL::SUM_ROWS; i += GQ_WARPS) sums[i * PL::SUM_PITCH + lane] = 0u; // afterwards whoever reads a sum clears it
  __syncthreads();

  // ---- this group's run of units ------------------------------------------------------------------
  const CacheView &c = a.c;
  const int dim = c.dim;
  const int items = a.heads_in_call * a.groups_per_head;
  const long long total = (long long)items * a.units;
  const int n_runs = (int)gridDim.x * GQ_GROUPS, run = (int)blockIdx.x * GQ_GROUPS + grp;
  auto run_begin = [&](int r) -> long long { return (long long)r * total / n_runs; };
  const long long u_begin = run_begin(run), u_end = run_begin(run + 1);

  int stage = 0;
  uint32_t phase = 0;
  auto wait_on = [&](uint64_t *bar, uint32_t parity) {
    if (*fail == 0 && !mbar_wait(bar, parity)) {
      *fail = 1;
      atomicExch(a.status, 1);
    }
    asm volatile("" ::: "memory"); // no read of what the barrier guards moves above the wait
  };

  if (producer) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GQ_REGS_PRODUCER));
    if (warp_all >= GQ_GROUPS * GQ_WARPS + GQ_GROUPS || lane != 0) return;
    griddep_wait(); // everything the cache holds is read through this thread's copies
    // The block must not end, nor a stage be written twice, while a copy is under way: once a wait has
    // given up nothing more is issued, and this thread leaves when every stage's latest copy has
    // landed (bounded; a stage that was never filled counts as landed).
    auto drain = [&]() {
      for (int s = 0; s < PL::STAGES; ++s)
        if (!mbar_wait(&full[s], s < stage ? phase : phase ^ 1u)) atomicExch(a.status, 1);
    };
    for (long long u = u_begin; u < u_end;) {
      const int item = (int)(u / a.units), u0 = (int)(u % a.units);
      const int cnt_u = (int)min((long long)(a.units - u0), u_end - u);
      u += cnt_u;
      const int h = a.head0 + item / a.groups_per_head;
      const int t0 = u0 * a.unit_tokens, t1 = min(a.n, (u0 + cnt_u) * a.unit_tokens);
      const uint8_t *kb = c.k_slab + (size_t)h * c.k_stride, *vb = c.v_slab + (size_t)h * c.v_stride;
      const float *ksb = c.k_scale + (size_t)h * c.s_stride;
      const uint8_t *vsb = reinterpret_cast<const uint8_t *>(c.v_scale + (size_t)h * c.s_stride);
      for (int c0 = t0; c0 < t1; c0 += CHUNK) {
        const int c1 = min(t1, c0 + CHUNK);
        // per chunk: the K rows with their scales, the V scales in one stage, the V rows
        for (int pass = 0; pass < 3; ++pass) {
          const int rowb = pass == 0 ? PL::KROW : pass == 1 ? 4 : PL::VROW;
          const int tn = pass == 0 ? PL::TKN : pass == 1 ? CHUNK : PL::TVN;
          const uint8_t *src = pass == 0 ? kb : pass == 1 ? vsb : vb;
          for (int t = c0; t < c1; t += tn) {
            wait_on(&empty[stage], phase ^ 1u);
            if (*fail != 0) { drain(); return; }
            const int cnt = min(tn, c1 - t);
            // sizes rounded up to 16 bytes run into the slack behind a head's rows and scales, never past it
            const uint32_t bytes = ((uint32_t)(cnt * rowb) + 15u) & ~15u;
            const uint32_t sbytes = pass ? 0u : (((uint32_t)cnt * 4u + 15u) & ~15u);
            if (!AQ_CHECK(a.status, (size_t)t * rowb + bytes <= (pass == 0 ? c.k_stride : pass == 1 ? (size_t)c.s_stride * 4 : c.v_stride) &&
                                        h >= 0 && h < c.n_heads, 13)) {
              *fail = 1; // consumers stop waiting; the block drains
              drain();
              return;
            }
            mbar_expect_tx(&full[stage], bytes + sbytes);
            bulk_g2s(stage_ptr(stage), src + (size_t)t * rowb, bytes, &full[stage]);
            if (sbytes) bulk_g2s(stage_ptr(stage) + GQ_STAGE, ksb + t, sbytes, &full[stage]);
            if (++stage == PL::STAGES) { stage = 0; phase ^= 1u; }
          }
        }
      }
    }
    drain();
    return;
  }

  // ======================= consumer warps ===========================================================
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(GQ_REGS_CONSUMER));
  const int gid = lane >> 2, tig = lane & 3;
  const uint32_t lane_table = table_addr | (uint32_t)(lane << 2);
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(GQ_GROUP_THREADS) : "memory"); };
  // The stages alternate between two teams of four warps (a stage is more work per warp, and the
  // teams overlap); every warp follows the sequence, `turn` says whose stage the current one is.
  const int team = warp >> 2, tw = warp & 3;
  int turn = 0;
  auto wait_full = [&]() { wait_on(&full[stage], phase); };
  auto release = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stage]);
  };
  auto next_stage = [&]() {
    turn ^= 1;
    if (++stage == PL::STAGES) { stage = 0; phase ^= 1u; }
  };
  const float isp = 1.f / sqrtf((float)P);
  const float attn_s = 1.f / (sqrtf((float)dim) * (float)P);
  // V stream roles: coordinates 64*half + 8*gid .. +7 of the tokens of every VTW-th 32-token group of the team's stages
  constexpr int HALVES = P / 64, VTW = 4 / HALVES;
  const int half = tw / VTW, vtw = tw % VTW, vunit = half * 8 + gid;
  const uint32_t usel = VB == 2 ? ((vunit & 1) ? 0x7362u : 0x5140u)
                                : (3 * vunit & 3) == 0 ? 0x0012u : (3 * vunit & 3) == 1 ? 0x0123u : (3 * vunit & 3) == 2 ? 0x0234u : 0x0345u;
  // softmax roles: WPQ warps per query slot
  constexpr int WPQ = GQ_WARPS / NQ, QPT = CHUNK / 4 / (WPQ * 32);
  constexpr int APT = (P * NQ + GQ_GROUP_THREADS - 1) / GQ_GROUP_THREADS; // running accumulators per thread
  const int sq = warp / WPQ, sthr = (warp % WPQ) * 32 + lane;

  for (long long u = u_begin; u < u_end;) {
    const int item = (int)(u / a.units), u0 = (int)(u % a.units);
    const int cnt_u = (int)min((long long)(a.units - u0), u_end - u);
    const long long item_first = (long long)item * a.units;
    u += cnt_u;
    const int hl = item / a.groups_per_head, qg = item % a.groups_per_head;
    const int q_first = qg * a.per_group, nq_here = min(a.per_group, a.nq - q_first);
    const int hq0 = hl * a.nq + q_first;
    const uint32_t *sg = c.signs + (size_t)(a.head0 + hl) * c.sign_words;
    const int t0 = u0 * a.unit_tokens, t1 = min(a.n, (u0 + cnt_u) * a.unit_tokens);

    // ---- rotate the queries (attention.cpp:537-550) and make them 31-bit fixed point -----------------
    if (warp < NQ) {
      float v[EPL];
      float part = 0.f, big = 0.f;
      const float *qp = a.q + (size_t)(hq0 + warp) * dim;
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        v[e] = (warp < nq_here && EPL * lane + e < dim) ? __ldg(qp + EPL * lane + e) : 0.f;
        part += v[e] * v[e];
      }
      const float qn = sqrtf(warp_sum(part) + 1e-12f);
      const float inv = 1.f / qn;
#pragma unroll
      for (int e = 0; e < EPL; ++e) v[e] = v[e] * inv * sign_of(sg, EPL * lane + e);
      warp_butterflies<EPL>(v, lane);
#pragma unroll
      for (int e = 0; e < EPL; ++e) big = fmaxf(big, fabsf(v[e]));
      big = warp_max(big);
      // |v| <= big < 2^(x+1): v * 2^(29-x) is below 2^30, and the scaling rounds nothing
      const int shift = big > 0.f && big < INFINITY ? 29 - ilogbf(big) : 0;
      const float up = ldexpf(1.f, shift >> 1), up2 = ldexpf(1.f, shift - (shift >> 1)); // 2^shift itself may not be a float
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        const uint32_t f = (uint32_t)__float2int_rn(v[e] * up * up2);
        qd[warp * P + EPL * lane + e] = (int)((f + 0x00808080u) ^ 0x00808080u); // bytes = signed digits, base 256
      }
      // a query that holds an infinity or a NaN makes every logit NaN, as its rotation would
      if (lane == 0) qscale[warp] = ldexpf(qn * 256e-4f * attn_s, -shift) * (qn < INFINITY ? 1.f : __int_as_float(0x7fc00000));
    }
    group_sync();
    // B operands of the K stream, one word per lane.  Column gid = (query 2*nt + (gid >> 2), place k = gid & 3):
    // sums of weight 256^(k+1), to which the high plane brings digit k and the low plane digit k + 1.
    // (The lowest place, low plane times digit 0, is below 2^-26 of the sum and left out.)
    for (int r = warp; r < PL::BQ_ROWS; r += GQ_WARPS) {
      const int nt = r / KR, i = r % KR, k = gid & 3;
      const uint32_t *qrow = reinterpret_cast<const uint32_t *>(qd) + (2 * nt + (gid >> 2)) * P;
      uint32_t x;
      if constexpr (KB == 4) {
        x = __byte_perm(qrow[k_coord<4, P>(tig, i, 0)] >> (8 * k), qrow[k_coord<4, P>(tig, i, 2)] >> (8 * k), 0x5410);
      } else {
        const int d = k + (i & 1); // one digit of four coordinates; there is no digit 4
        const uint32_t pick = (uint32_t)(d & 3) | ((uint32_t)(4 + (d & 3)) << 4);
        const uint32_t y = prmt_sel(qrow[k_coord<KB, P>(tig, i, 0)], qrow[k_coord<KB, P>(tig, i, 1)], pick);
        const uint32_t z = prmt_sel(qrow[k_coord<KB, P>(tig, i, 2)], qrow[k_coord<KB, P>(tig, i, 3)], pick);
        x = d < 4 ? __byte_perm(y, z, 0x5410) : 0u;
      }
      bqs[r * 32 + lane] = x;
    }
    group_sync();
    float acc_run[APT];
#pragma unroll
    for (int r = 0; r < APT; ++r) acc_run[r] = 0.f;

    for (int c0 = t0; c0 < t1; c0 += CHUNK) {
      const int len = min(t1 - c0, CHUNK);
      const bool first = c0 == t0;
      // ---- K stream: logits into sc[query][token] ---------------------------------------------------
      uint32_t bq[NT][KR];
      float qs[NT], lane_max[NT];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int i = 0; i < KR; ++i) bq[nt][i] = bqs[(nt * KR + i) * 32 + lane];
        qs[nt] = qscale[2 * nt + (tig >> 1)];
        lane_max[nt] = -1e30f; // where upstream's running maximum starts (attention.cpp:384)
      }
      for (int t = 0; t < len; t += PL::TKN) {
        if (turn != team) { next_stage(); continue; }
        wait_full();
        const uint8_t *st = stage_ptr(stage);
        const float *ksc = reinterpret_cast<const float *>(st + GQ_STAGE);
        // tiles of 16 tokens; rows past the chunk's end are scored too (they index nothing) and not stored
#pragma unroll(PL::TKN / 64 <= 2 ? 2 : 1)
        for (int m = 0; m < PL::TKN / 64; ++m) {
          const int mt = tw * (PL::TKN / 64) + m;
          int d[NT][4];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) d[nt][r] = 0;
          uint32_t w0[KLane<KB, P>::WORDS], w1[KLane<KB, P>::WORDS];
          load_k_lane<KB, P>(st + (size_t)(mt * 16 + gid) * PL::KROW, tig, w0);
          load_k_lane<KB, P>(st + (size_t)(mt * 16 + gid + 8) * PL::KROW, tig, w1);
          const int own = mt * 16 + gid + 8 * (tig & 1); // the token whose logits this lane ends up with
          const float ks = ksc[own];
          uint32_t a0[KR], a1[KR];
          expand_k<KB, P>(w0, tig, lane_table, a0);
          expand_k<KB, P>(w1, tig, lane_table, a1);
#pragma unroll
          for (int s = 0; s < KR; s += 2) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_s8s8(d[nt], a0[s], a1[s], a0[s + 1], a1[s + 1], bq[nt][s], bq[nt][s + 1]);
          }
          // this lane holds places 2*(tig & 1) and + 1 of query 2*nt + (tig >> 1), rows gid and gid + 8;
          // the other two places are in the neighbouring lane
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const float f0 = (float)(d[nt][1] * 256 + d[nt][0]), f1 = (float)(d[nt][3] * 256 + d[nt][2]);
            const bool odd = (tig & 1) != 0;
            const float got = __shfl_xor_sync(0xffffffffu, odd ? f0 : f1, 1);
            const float sum = odd ? fmaf(f1, 65536.f, got) : fmaf(got, 65536.f, f0);
            const float logit = sum * qs[nt] * ks;
            if (t + own < len) {
              sc[(2 * nt + (tig >> 1)) * PL::SCORE_PITCH + t + own] = logit;
              lane_max[nt] = fmaxf(lane_max[nt], logit);
            }
          }
        }
        release();
        next_stage();
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        float m = lane_max[nt];
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((lane & 0x1d) == 0) red[(2 * nt + (tig >> 1)) * 8 + warp] = m; // lanes 0 and 2
      }
      group_sync();
      // ---- exact softmax of the chunk; thread `sthr` of query slot sq owns quads of four tokens ------------
      float mx = red[sq * 8];
#pragma unroll
      for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red[sq * 8 + w]);
      float e4[QPT][4];
      float ls = 0.f, wsum = 0.f;
      wait_full();
      {
        const float4 *vs4 = reinterpret_cast<const float4 *>(stage_ptr(stage));
        const float4 *sc4 = reinterpret_cast<const float4 *>(sc + sq * PL::SCORE_PITCH);
#pragma unroll
        for (int r = 0; r < QPT; ++r) {
          const int qi = r * (WPQ * 32) + sthr;
          if (4 * qi < len) {
            const float4 s4 = sc4[qi], v4 = vs4[qi];
            const float sv[4] = {s4.x, s4.y, s4.z, s4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const bool live = 4 * qi + k < len; // padding weighs nothing
              const float e = live ? exp_nonpos(sv[k] - mx) : 0.f;
              ls += e;
              e4[r][k] = live ? e * vv[k] * isp : 0.f;
              wsum += e4[r][k];
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) e4[r][k] = 0.f;
          }
        }
      }
      ls = warp_sum(ls);
      wsum = warp_sum(wsum);
      if (lane == 0) { red_l[warp] = ls; red_w[warp] = wsum; }
      group_sync(); // every score is in registers (the weights may take their place), every V scale has been read
      if (turn == team) release();
      next_stage();
      ls = wsum = 0.f;
#pragma unroll
      for (int w = 0; w < WPQ; ++w) { ls += red_l[sq * WPQ + w]; wsum += red_w[sq * WPQ + w]; }
      // weights -> fixed point with the chunk's total mapped to 2^30; a total that is NaN or
      // infinite (a NaN logit, an infinite V scale) makes the accumulator NaN, as floating-point sums would be
      const float fx = (wsum > 0.f && wsum < INFINITY) ? 1073741824.0f / wsum : 0.f;
      const float inv_fx = fx > 0.f ? wsum * (1.0f / 1073741824.0f) : (wsum == 0.f ? 0.f : __int_as_float(0x7fc00000));
      uint32_t wint = 0u;
#pragma unroll
      for (int r = 0; r < QPT; ++r) {
        const int qi = r * (WPQ * 32) + sthr;
        if (4 * qi < ((len + 31) & ~31)) {
          uint32_t f[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) { f[k] = __float2uint_rn(e4[r][k] * fx); wint += f[k]; }
          const uint32_t a01 = __byte_perm(f[0], f[1], 0x5140), a23 = __byte_perm(f[2], f[3], 0x5140);
          const uint32_t b01 = __byte_perm(f[0], f[1], 0x7362), b23 = __byte_perm(f[2], f[3], 0x7362);
          const uint32_t dg[4] = {__byte_perm(a01, a23, 0x5410), __byte_perm(a01, a23, 0x7632),
                                  __byte_perm(b01, b23, 0x5410), __byte_perm(b01, b23, 0x7632)};
          // quad qi = (group of 32, set of 16, lane tg): beside its other set; the four tokens start
          // with number tg of the quad, the order in which lane tg of the V stream reads the rows
          const int tg = qi & 3, pos = (qi >> 3) * 8 + tg * 2 + ((qi >> 2) & 1);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            wd[(sq * 4 + k) * PL::W_PITCH + pos] = __funnelshift_r(dg[k], dg[k], 8 * tg);
        }
      }
      if constexpr (VB == 2) {
        wint = __reduce_add_sync(0xffffffffu, wint);
        if (lane == 0) wtot[warp] = wint;
      }
      if (warp % WPQ == 0 && lane == 0) { // the segment's running maximum and sum
        const float m_old = first ? mx : s_m[sq], m_new = fmaxf(m_old, mx);
        const float alpha = first ? 0.f : expf(m_old - m_new), beta = expf(mx - m_new);
        s_l[sq] = (first ? 0.f : s_l[sq] * alpha) + ls * beta;
        s_m[sq] = m_new;
        s_alpha[sq] = alpha;
        s_scale[sq] = beta * inv_fx * (VB == 2 ? 1e-4f : 256e-4f);
      }
      group_sync();
      // ---- V stream: coordinates x weights -------------------------------------------------------------
      int dv[4][PL::PLANES][NT][4]; // [coordinate pair][plane][nt][.]
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int pl = 0; pl < PL::PLANES; ++pl)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) dv[i][pl][nt][r] = 0;
      for (int t = 0; t < len; t += PL::TVN) {
        if (turn != team) { next_stage(); continue; }
        wait_full();
        const uint8_t *st = stage_ptr(stage);
#pragma unroll 1
        for (int g32 = vtw; g32 < PL::TVN / 32; g32 += VTW) {
          if (t + g32 * 32 >= len) break;
          uint32_t x[2][4];
#pragma unroll
          for (int set = 0; set < 2; ++set) {
            uint32_t w[4][VWords<VB>::N];
#pragma unroll
            for (int j = 0; j < 4; ++j) // token 4*tig + (j + tig) mod 4: the lanes of a load read different banks
              load_v_unit<VB, P>(st + (size_t)(g32 * 32 + set * 16 + 4 * tig + ((j + tig) & 3)) * PL::VROW, vunit, w[j]);
            gather_v<VB>(w, usel, x[set]);
          }
          // column gid = (query, place k): digit k of the two sets' weights, and digit k + 1 (none above 3)
          uint2 wk[NT], wn[NT];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const uint32_t *wp = wd + (nt * 8 + gid) * PL::W_PITCH + ((t >> 5) + g32) * 8 + tig * 2;
            wk[nt] = *reinterpret_cast<const uint2 *>(wp);
            if constexpr (VB != 2) wn[nt] = (gid & 3) == 3 ? make_uint2(0u, 0u) : *reinterpret_cast<const uint2 *>(wp + PL::W_PITCH);
            if constexpr (VB == 4) { // {k, k+1} digits of tokens 0, 1 | of tokens 2, 3
              const uint2 p = wk[nt], q = wn[nt];
              wk[nt] = make_uint2(__byte_perm(p.x, q.x, 0x5140), __byte_perm(p.x, q.x, 0x7362));
              wn[nt] = make_uint2(__byte_perm(p.y, q.y, 0x5140), __byte_perm(p.y, q.y, 0x7362));
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t ua[2], va[2], ub[2], vb[2];
            plane_pair<VB>(x[0], i, lane_table, ua, va);
            plane_pair<VB>(x[1], i, lane_table, ub, vb);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              if constexpr (VB == 2) { // both bits against the weight's digits, in sums of their own
                mma_u8u8(dv[i][1][nt], ua[0], ua[1], ub[0], ub[1], wk[nt].x, wk[nt].y);
                mma_u8u8(dv[i][0][nt], va[0], va[1], vb[0], vb[1], wk[nt].x, wk[nt].y);
              } else if constexpr (VB == 3) { // high planes against digit k, low planes against digit k + 1
                mma_s8u8(dv[i][0][nt], ua[0], ua[1], ub[0], ub[1], wk[nt].x, wk[nt].y);
                mma_s8u8(dv[i][0][nt], va[0], va[1], vb[0], vb[1], wn[nt].x, wn[nt].y);
              } else {
                mma_s8u8(dv[i][0][nt], ua[0], ua[1], va[0], va[1], wk[nt].x, wk[nt].y);
                mma_s8u8(dv[i][0][nt], ub[0], ub[1], vb[0], vb[1], wn[nt].x, wn[nt].y);
              }
            }
          }
        }
        release();
        next_stage();
      }
      // the warps that shared the coordinates add up: sums[half][coordinate][plane][nt][column & 1][tig][gid]
      {
        const uint32_t sa = smem_u32(sums) + (uint32_t)(half * (PL::SUM_ROWS / HALVES) * PL::SUM_PITCH + tig * 8 + gid) * 4u;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int pl = 0; pl < PL::PLANES; ++pl)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
              for (int r = 0; r < 4; ++r)
                red_shared_add(sa + (uint32_t)((((2 * i + (r >> 1)) * PL::PLANES + pl) * NT + nt) * 2 + (r & 1)) * (PL::SUM_PITCH * 4u),
                               (uint32_t)dv[i][pl][nt][r]);
      }
      group_sync();
      // ---- exact totals per (query, coordinate), scaled onto the running accumulator -------------------
#pragma unroll
      for (int r = 0; r < APT; ++r) {
        const int e = gtid + r * GQ_GROUP_THREADS; // bits: unit 3, query & 1, coordinate 3, half, nt
        if (e >= P * NQ) break;
        const int un = e & 7, qp = (e >> 3) & 1, co = (e >> 4) & 7, rest = e >> 7;
        const int hf = rest % HALVES, nt = rest / HALVES, qq = 2 * nt + qp;
        long long s[PL::PLANES];
#pragma unroll
        for (int pl = 0; pl < PL::PLANES; ++pl) {
          uint32_t *p = sums + ((((hf * 8 + co) * PL::PLANES + pl) * NT + nt) * 2) * PL::SUM_PITCH + qp * 16 + un;
          const int d0 = (int)p[0], d1 = (int)p[PL::SUM_PITCH], d2 = (int)p[8], d3 = (int)p[PL::SUM_PITCH + 8]; // place = 2*(tig & 1) + (column & 1)
          p[0] = p[PL::SUM_PITCH] = p[8] = p[PL::SUM_PITCH + 8] = 0u;
          s[pl] = ((long long)d3 * 256 + d2) * 65536 + ((long long)d1 * 256 + d0);
        }
        long long tot = s[0];
        if constexpr (VB == 2) { // centroid*10^4 = -15104 + 19632*(high bit) + 10576*(low bit)
          uint32_t wt = 0u;
#pragma unroll
          for (int w = 0; w < WPQ; ++w) wt += wtot[qq * WPQ + w];
          tot = 19632 * (s[1] >> (7 - 2 * (co & 3))) + 10576 * (s[0] >> (6 - 2 * (co & 3))) - 15104ll * wt;
        }
        const float x = (float)tot * s_scale[qq];
        acc_run[r] = first ? x : acc_run[r] * s_alpha[qq] + x;
      }
    }
    // ---- hand the segment's accumulators to one warp per query ----------------------------------------------
#pragma unroll
    for (int r = 0; r < APT; ++r) {
      const int e = gtid + r * GQ_GROUP_THREADS;
      if (e >= P * NQ) break;
      const int un = e & 7, qp = (e >> 3) & 1, co = (e >> 4) & 7, rest = e >> 7;
      accb[(2 * (rest / HALVES) + qp) * P + (rest % HALVES) * 64 + un * 8 + co] = acc_run[r];
    }
    group_sync();
    if (warp < nq_here) {
      const int hq = hq0 + warp;
      float v[EPL];
#pragma unroll
      for (int e = 0; e < EPL; ++e) v[e] = accb[warp * P + EPL * lane + e];
      float L = s_l[warp];
      bool done = true;
      if (cnt_u != a.units) { // other groups hold the rest of this item
        const int r_first = (int)(((item_first + 1) * n_runs - 1) / total), r_last = (int)(((item_first + a.units) * n_runs - 1) / total);
        const int parts = r_last - r_first + 1;
        auto piece = [&](int p) { // a head's later pieces start their runs; its first one may not
          const int second = p == 0 && run_begin(r_first) < item_first ? 1 : 0;
          return a.partial + ((size_t)(2 * (r_first + p) + second) * a.per_group + warp) * (2 + P);
        };
        float *pp = piece(run - r_first);
        if (!AQ_CHECK(a.status, r_first >= 0 && r_last < n_runs && run >= r_first && run <= r_last && hq >= 0 &&
                                    hq < a.heads_in_call * a.nq && warp < a.per_group, 14)) continue;
        if (lane == 0) { pp[0] = s_m[warp]; pp[1] = L; }
#pragma unroll
        for (int e = 0; e < EPL; ++e) pp[2 + EPL * lane + e] = v[e];
        __threadfence();
        __syncwarp();
        int ticket = 0;
        if (lane == 0) ticket = atomicAdd(&a.counters[hq], 1);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        done = ticket == parts - 1;
        if (done) { // the last to arrive merges; NaN sums and zero weights travel as they do upstream
          if (lane == 0) a.counters[hq] = 0;
          __threadfence();
          float M = -INFINITY;
          for (int p = lane; p < parts; p += 32) M = fmaxf(M, __ldcg(piece(p)));
          M = warp_max(M);
          L = 0.f;
#pragma unroll
          for (int e = 0; e < EPL; ++e) v[e] = 0.f;
#pragma unroll 4
          for (int p = 0; p < parts; ++p) {
            const float *row = piece(p);
            const float w = expf(__ldcg(row) - M);
            L += __ldcg(row + 1) * w;
#pragma unroll
            for (int e = 0; e < EPL; ++e) v[e] += w * __ldcg(row + 2 + EPL * lane + e);
          }
        }
      }
      if (done) { // normalise, inverse transform (core/fwht.cpp:106-134), store
        const float invl = 1.f / L;
#pragma unroll
        for (int e = 0; e < EPL; ++e) v[e] *= invl;
        warp_butterflies<EPL>(v, lane);
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          const int j = EPL * lane + e;
          if (j < dim) a.out[(size_t)hq * dim + j] = v[e] * isp * sign_of(sg, j);
        }
      }
    }
  }
}

} // namespace aq
