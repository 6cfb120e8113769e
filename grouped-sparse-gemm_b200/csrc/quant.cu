// Activation quantizers: bf16 -> e2m1 codes + one UE4M3 scale per 32 elements, written straight
// into the grouped GEMM's B-operand layouts (row-major codes, swizzled scale atoms).
//
// quant_act, silu_mul_quant_act and scatter_quant_act_planned share two kernels.  Their work is the live rows
// (r < counts[e]) of the batched operand, found through a prefix sum of counts that every block makes for itself, so that
// skewed or mostly empty capacities cost nothing.  One whole 32-element K-block per lane (64 bytes in, or 128 with gate and
// up; 16 bytes of codes out; the scale step, with its two IEEE divisions, once per block).  With long rows
// (quant_batched_kernel) a warp takes a row, or a piece of one where there are fewer rows than warps, 32 K-blocks at a
// time; otherwise (quant_quads_kernel) the rows' K-blocks are laid end to end and dealt four by four, so that short rows
// and remainders leave no lane idle.  The bytes of the scale buffer that no live row writes become 0x38 in the same kernel,
// a 16-byte line per thread.
// Bound: HBM for plain rows (131072 rows of 2048: 118 us, 687 MB), issue slots (0.68 of them used) and L2 for gathered
// ones (102 us; 150 MB written, the rows read from L2 eight times over), the special-function unit and issue for SiTU.
// Loads are 32 bytes a lane where the input is aligned to that: 16-byte loads at a stride of 64 bytes take twice the
// passes through L1.  A warp per 16-byte line of the scale buffer, dead lines included, took 466 us for 32768 live rows of
// 3072 (SiTU) in a capacity of 524288 where the row form takes 172, and 82 us for the gather of those rows where it takes 40.
//
// scatter_quant_act is driven by a flat routing list instead (source token -> destination row), so its scale buffer is
// pre-filled with a memset node.
#include "common.cuh"

namespace pnv {
namespace {

constexpr int kThreads = 256;
constexpr int kWarpsPerBlock = kThreads / 32;

// Four adjacent lanes hold the scale bytes of four consecutive K-blocks; lane 4j returns their word.
__device__ __forceinline__ uint32_t gather_sf_word(uint32_t my_byte) {
  return my_byte | (__shfl_down_sync(0xffffffffu, my_byte, 1) << 8) |
         (__shfl_down_sync(0xffffffffu, my_byte, 2) << 16) | (__shfl_down_sync(0xffffffffu, my_byte, 3) << 24);
}

// One 32-element block in one lane: 64 bytes in, two bf16 to a register.  `wide`: the source is 32-byte aligned.  (The load
// is volatile with a memory clobber so that the compiler keeps it behind pdl_wait().)
struct BlockRegs {
  uint32_t lo[8], hi[8];
};
__device__ __forceinline__ void load32(const uint8_t* src, bool wide, uint32_t (&w)[8]) {
  if (wide) {
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "l"(src) : "memory");
  } else {
    const uint4 v0 = __ldg(reinterpret_cast<const uint4*>(src)), v1 = __ldg(reinterpret_cast<const uint4*>(src) + 1);
    w[0] = v0.x; w[1] = v0.y; w[2] = v0.z; w[3] = v0.w;
    w[4] = v1.x; w[5] = v1.y; w[6] = v1.z; w[7] = v1.w;
  }
}
__device__ __forceinline__ void load_block(const uint8_t* src, bool wide, BlockRegs& b) {
  load32(src, wide, b.lo);
  load32(src + 32, wide, b.hi);
}
__device__ __forceinline__ float block_amax(const BlockRegs& b) {
  const uint32_t m = bf16x2_max(bf16x2_amax8(b.lo), bf16x2_amax8(b.hi));
  return fmaxf(fmaxf(bf16_lo(m), bf16_hi(m)), 0.f);       // (a NaN counts as nothing)
}
__device__ __forceinline__ uint4 block_codes(const BlockRegs& b, float inv) {
  return make_uint4(quant8_packed(b.lo[0], b.lo[1], b.lo[2], b.lo[3], inv), quant8_packed(b.lo[4], b.lo[5], b.lo[6], b.lo[7], inv),
                    quant8_packed(b.hi[0], b.hi[1], b.hi[2], b.hi[3], inv), quant8_packed(b.hi[4], b.hi[5], b.hi[6], b.hi[7], inv));
}
__device__ __forceinline__ void store_codes(uint4* dst, const uint4& codes, bool dst16) {      // 8-byte aligned otherwise
  if (dst16) {
    *dst = codes;
  } else {
    reinterpret_cast<uint2*>(dst)[0] = make_uint2(codes.x, codes.y);
    reinterpret_cast<uint2*>(dst)[1] = make_uint2(codes.z, codes.w);
  }
}
// Every value times the bf16 weight w, rounded to bf16 (the product of two bf16 numbers is exact in float, so the packed
// multiplication rounds like the float product rounded to bf16).
__device__ __forceinline__ void block_weight(BlockRegs& b, float w) {
  const __nv_bfloat162 w2 = __float2bfloat162_rn(w);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    b.lo[i] = as_u32(__hmul2(as_bf162(b.lo[i]), w2));
    b.hi[i] = as_u32(__hmul2(as_bf162(b.hi[i]), w2));
  }
}

// Where a row's values come from.
//   kPlain   the row itself, x is [E, cap, K]
//   kGated   x is [E, cap, 2K] holding gate and up; the gated activation is applied first
//   kGather  row src_tok[slot] of x [T, K], optionally times the router weight of routing src_route[slot]
enum RowSource : int { kPlain = 0, kGated = 1, kGather = 2 };

// 32 K-blocks from kb0 on, one per lane in b, are scaled, rounded and stored; a row's four scales of one 128-K group are one
// aligned word of the swizzled layout.  KB: the blocks of the whole row.
__device__ __forceinline__ void finish_blocks(const BlockRegs& b, int kb0, int KB, float gs, uint4* __restrict__ dst,
                                              uint8_t* __restrict__ sf_row, int lane) {
  const int kb = kb0 + lane;
  uint32_t sf_byte = kBenignSf;   // blocks past K keep the benign byte in the layout's slop
  if (kb < KB) {
    float inv;
    block_scale(block_amax(b), gs, sf_byte, inv);
    dst[kb] = block_codes(b, inv);
  }
  const uint32_t word = gather_sf_word(sf_byte);
  if ((lane & 3) == 0 && kb < KB) *reinterpret_cast<uint32_t*>(sf_row + (kb >> 2) * 512) = word;
}

// scatter_quant_act: one warp per routing of the flat plan.
__global__ void __launch_bounds__(kThreads)
scatter_quant_kernel(const __nv_bfloat16* __restrict__ a1, const long long* __restrict__ flat_tok,
                     const long long* __restrict__ dest_global, const float* __restrict__ topk_w,
                     const float* __restrict__ gscale, int gscale_per_expert, unsigned n_routes,
                     int K, int E, int cap, uint8_t* __restrict__ b_act, uint8_t* __restrict__ sfb) {
  pdl_wait();
  pdl_launch_dependents();
  const int KB = K / kSfBlock;
  const int n_rt = sf_row_atoms(cap);
  const int n_kt = sf_k_atoms(K);
  const long long trash = (long long)E * cap;
  const bool wide = (reinterpret_cast<uintptr_t>(a1) & 31) == 0;
  const int lane = threadIdx.x & 31;
  const unsigned warp0 = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  const unsigned nwarps = gridDim.x * kWarpsPerBlock;
  for (unsigned i = warp0; i < n_routes; i += nwarps) {
    const long long dest = dest_global[i];
    if (dest == trash) continue;   // dropped routing: non-local expert or past capacity
    const int e = (int)((unsigned)dest / (unsigned)cap);     // dest < E * cap < 2^31
    const int r = (int)dest - e * cap;
    const float gs = gscale_per_expert ? gscale[e] : gscale[0];
    const bool weighted = topk_w != nullptr;
    const float w = weighted ? __bfloat162float(__float2bfloat16_rn(topk_w[i])) : 1.f;
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a1 + flat_tok[i] * K);
    for (int kb0 = 0; kb0 < KB; kb0 += 32) {
      BlockRegs b;
      if (kb0 + lane < KB) load_block(src + 64LL * (kb0 + lane), wide, b);
      if (weighted) block_weight(b, w);
      finish_blocks(b, kb0, KB, gs, reinterpret_cast<uint4*>(b_act + dest * (K / 2)), sfb + sf_offset(e, r, 0, n_rt, n_kt), lane);
    }
  }
}

// One word of scales.
__device__ __forceinline__ void store_sf_word(uint8_t* dst, uint32_t w, bool dst4) {
  if (dst4) {
    *reinterpret_cast<uint32_t*>(dst) = w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = (uint8_t)(w >> (8 * i));
  }
}

// Every byte of a scale buffer that no live row (r < counts[e]) writes becomes 0x38: whole 16-byte lines behind which
// no row is live, single words of the others.  (K-block slop of a live row is part of the words that row writes.)  The
// kernels that place rows do this themselves, each thread a share of the lines: as a memset in front of them it was a
// launch of its own and kept them from starting while their predecessor drains.  (kLoose: the buffer may be less than
// 16-byte aligned, and is then filled word by word, or byte by byte.)
template <bool kLoose>
__device__ __forceinline__ void benign_fill_dead(const int* __restrict__ counts, int E, int cap, int n_rt, int n_kt,
                                                 uint8_t* __restrict__ sfb) {
  const uint32_t w4 = kBenignSf * 0x01010101u;
  const unsigned lines = (unsigned)E * n_rt * n_kt * 32u;
  const bool sfb16 = !kLoose || (reinterpret_cast<uintptr_t>(sfb) & 15) == 0;
  const bool sfb4 = !kLoose || (reinterpret_cast<uintptr_t>(sfb) & 3) == 0;
  for (unsigned c = blockIdx.x * kThreads + threadIdx.x; c < lines; c += gridDim.x * kThreads) {
    const unsigned a_kt = (c >> 5) / (unsigned)n_kt;
    const unsigned e = a_kt / (unsigned)n_rt;
    const int r0 = (int)(a_kt - e * (unsigned)n_rt) * 128 + (int)(c & 31);
    const int cnt = min(counts[e], cap);
    uint8_t* line = sfb + (long long)c * 16;
    if (r0 >= cnt && sfb16) {
      *reinterpret_cast<uint4*>(line) = make_uint4(w4, w4, w4, w4);
    } else {
#pragma unroll
      for (int g = 0; g < 4; ++g)
        if (r0 + 32 * g >= cnt) store_sf_word(line + 4 * g, w4, sfb4);
    }
  }
}

// The same for the kernel that copies rows: neighbouring atoms of a row atom per warp, up to eight where every warp has as
// many to do, so that the divisions and the count serve eight stores a lane.  (2048 experts x 4 rows x 7168: 28 us with a
// line per thread, 23 so.  The quantizers' small calls are a microsecond faster with a line per thread.)
__device__ __forceinline__ void benign_fill_dead_atoms(const int* __restrict__ counts, int E, int cap, int n_rt, int n_kt,
                                                       uint8_t* __restrict__ sfb) {
  const uint32_t w4 = kBenignSf * 0x01010101u;
  const bool sfb16 = (reinterpret_cast<uintptr_t>(sfb) & 15) == 0, sfb4 = (reinterpret_cast<uintptr_t>(sfb) & 3) == 0;
  const unsigned nwarps = gridDim.x * kWarpsPerBlock, lane = threadIdx.x & 31;
  const unsigned per_unit = min(8u, max(1u, (unsigned)E * n_rt * n_kt / nwarps));
  const unsigned n_kc = ((unsigned)n_kt + per_unit - 1) / per_unit, units = (unsigned)E * n_rt * n_kc;
  for (unsigned u = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < units; u += nwarps) {
    const unsigned row_atom = u / n_kc, kt0 = (u - row_atom * n_kc) * per_unit, e = row_atom / (unsigned)n_rt;
    const int base = (int)(row_atom - e * (unsigned)n_rt) * 128, r0 = base + (int)lane, cnt = min(counts[e], cap);
    if (cnt - base >= 128) continue;                      // (every row of these atoms is live)
    const unsigned n = min(per_unit, (unsigned)n_kt - kt0);
    uint8_t* line = sfb + ((long long)row_atom * n_kt + kt0) * 512 + lane * 16;
    if (r0 >= cnt && sfb16) {
      for (unsigned i = 0; i < n; ++i) *reinterpret_cast<uint4*>(line + i * 512) = make_uint4(w4, w4, w4, w4);
    } else {
      for (unsigned i = 0; i < n; ++i) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
          if (r0 + 32 * g >= cnt) store_sf_word(line + i * 512 + 4 * g, w4, sfb4);
      }
    }
  }
}

// The live rows of a batched operand, numbered expert after expert.  make() builds the prefix sums of the clamped
// counts - up to 32 experts every warp in its own registers, without a barrier; up to kMaxPrefixExperts the block in
// shared memory - and find() turns a row's number into its slot.  With more experts there are no prefix sums: every slot is
// a row and the dead ones are skipped.  All lanes of a warp ask for the same row.  Row numbers are unsigned 32-bit: K = 32
// leaves room for more than 2^31 rows in this GPU's memory.
constexpr int kMaxPrefixExperts = 8192;
struct LiveRows {
  const int* counts;
  int E, cap;
  unsigned* prefix;      // shared memory, [E + 1]
  unsigned lane_first;   // up to 32 experts: first row of expert `lane` (the largest number past the last)
  unsigned total;
  __device__ __forceinline__ void make(const int* counts_, int E_, int cap_, unsigned* smem) {
    counts = counts_; E = E_; cap = cap_; prefix = smem; lane_first = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (E > kMaxPrefixExperts) { total = (unsigned)E * (unsigned)cap; return; }
    if (E <= 32) {
      const unsigned c = lane < E ? (unsigned)max(0, min(counts[lane], cap)) : 0u;
      unsigned v = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      lane_first = lane < E ? v - c : 0xFFFFFFFFu;
      total = __shfl_sync(0xffffffffu, v, 31);
      return;
    }
    // Every thread takes a run of counts (one up to 256 experts; otherwise they go through shared memory by independent
    // loads, and a run of odd length has no bank conflicts), the runs' sums are scanned over the block, and every thread
    // turns its run into prefix sums in place.  (256 counts at a time, a global load and two barriers each, took 7 us for
    // 4096 experts.)
    __shared__ unsigned s_warp[kWarpsPerBlock];
    auto count = [&](int e) { return (unsigned)max(0, min(counts[e], cap)); };
    const int run = ((E + kThreads - 1) / kThreads) | 1, lo = (int)threadIdx.x * run, hi = min(E, lo + run);
    unsigned sum = 0;
    if (run == 1) {
      if (lo < E) sum = count(lo);
    } else {
#pragma unroll 4
      for (int e = threadIdx.x; e < E; e += kThreads) smem[e + 1] = count(e);
      __syncthreads();
      for (int e = lo; e < hi; ++e) sum += smem[e + 1];
    }
    unsigned v = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) s_warp[warp] = v;
    __syncthreads();
    unsigned before = v - sum, all = 0;
#pragma unroll
    for (int i = 0; i < kWarpsPerBlock; ++i) {
      if (i < warp) before += s_warp[i];
      all += s_warp[i];
    }
    if (run == 1) {
      if (lo < E) smem[lo + 1] = before + sum;
    } else {
      for (int e = lo; e < hi; ++e) {
        before += smem[e + 1];
        smem[e + 1] = before;
      }
    }
    if (threadIdx.x == 0) smem[0] = 0;
    __syncthreads();
    total = all;
  }
  // row number j < total -> expert and row of the expert; false for a dead slot (only without prefix sums)
  __device__ __forceinline__ bool find(unsigned j, int& e, int& r) const {
    if (E <= 32) {       // the last expert whose first row is at or before j
      e = 31 - __clz(__ballot_sync(0xffffffffu, lane_first <= j));
      r = (int)(j - __shfl_sync(0xffffffffu, lane_first, e));
      return true;
    }
    if (E > kMaxPrefixExperts) {
      e = (int)(j / (unsigned)cap);
      r = (int)(j - (unsigned)e * (unsigned)cap);
      return r < counts[e];
    }
    int lo = 0, hi = E - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (prefix[mid] <= j) lo = mid;
      else hi = mid - 1;
    }
    e = lo;
    r = (int)(j - prefix[lo]);
    return true;
  }
  // The same for a row of each lane's own (all lanes take part); a dead slot's expert is -1.
  __device__ __forceinline__ void find_each(unsigned j, int& e, int& r) const {
    int lo = 0;
    if (E <= 32) {
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const unsigned first = __shfl_sync(0xffffffffu, lane_first, lo + step);      // (lo + step < 32)
        if (first <= j) lo += step;
      }
      r = (int)(j - __shfl_sync(0xffffffffu, lane_first, lo));
    } else if (E > kMaxPrefixExperts) {
      lo = (int)(j / (unsigned)cap);
      r = (int)(j - (unsigned)lo * (unsigned)cap);
      if (lo >= E || r >= counts[lo]) lo = -1;
    } else {
      int hi = E - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= j) lo = mid;
        else hi = mid - 1;
      }
      r = (int)(j - prefix[lo]);
    }
    e = lo;
  }
};
size_t live_rows_smem(int E) { return E <= 32 || E > kMaxPrefixExperts ? 0 : sizeof(int) * (size_t)(E + 1); }

struct RowsArgs {
  const __nv_bfloat16* x;
  const int* src_tok;
  const int* src_route;
  const float* topk_w;
  const float* gscale;
  const int* counts;
  uint8_t* b_act;
  uint8_t* sfb;
  GatedAct act;
  int gscale_per_expert, E, cap, K, interleaved;
  int filled;            // the scale buffer already holds the benign byte everywhere
};

// Blocks per SM: four hold 64 registers a thread; five or six spill (6 to 17 % slower with the activation), three with the
// next step's loads ahead of the arithmetic are 15 % slower.  The grid is one wave of them.
constexpr int kBatchedBlocks = 4;

// A warp takes a row, or a piece of one: for rows of many K-blocks, 16-byte aligned destinations.
template <int kSrc>
__global__ void __launch_bounds__(kThreads, kBatchedBlocks)
quant_batched_kernel(const RowsArgs a) {
  extern __shared__ unsigned s_prefix[];
  pdl_wait();
  pdl_launch_dependents();
  const int KB = a.K / kSfBlock;
  const int n_rt = sf_row_atoms(a.cap);
  const int n_kt = sf_k_atoms(a.K);
  const bool wide = (reinterpret_cast<uintptr_t>(a.x) & 31) == 0;
  const int lane = threadIdx.x & 31;
  LiveRows rows;
  rows.make(a.counts, a.E, a.cap, s_prefix);
  const unsigned nwarps = gridDim.x * kWarpsPerBlock;
  // With fewer rows than warps a row is cut into pieces of 32 K-blocks or more: a decode step then takes as long as one
  // piece.  (Consecutive warps take consecutive rows of one piece; the scale words of 32 rows share lines.)
  unsigned pieces = 1;
  int piece_blocks = KB;
  if (rows.total > 0 && rows.total <= nwarps / 2u && KB > 32) {
    pieces = min(nwarps / rows.total, (unsigned)(KB + 31) / 32u);
    piece_blocks = (int)(((unsigned)KB + pieces - 1) / pieces + 31) / 32 * 32;
    pieces = (unsigned)(KB + piece_blocks - 1) / (unsigned)piece_blocks;
  }
  const unsigned units = rows.total * pieces;
  const long long row_bytes = (kSrc == kGated ? 4LL : 2LL) * a.K;
  for (unsigned u = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); u < units; u += nwarps) {
    const unsigned piece = pieces > 1 ? u / rows.total : 0u;
    int e, r;
    if (!rows.find(u - piece * rows.total, e, r)) continue;
    const long long slot = (long long)e * a.cap + r;
    const int lo = (int)piece * piece_blocks, hi = min(KB, lo + piece_blocks);
    const float gs = a.gscale_per_expert ? a.gscale[e] : a.gscale[0];
    const bool weighted = kSrc == kGather && a.topk_w != nullptr;
    float w = 1.f;
    long long src_row = slot;
    if constexpr (kSrc == kGather) {
      src_row = a.src_tok[slot];
      if (weighted) w = __bfloat162float(__float2bfloat16_rn(a.topk_w[a.src_route[slot]]));
    }
    const uint8_t* src = reinterpret_cast<const uint8_t*>(a.x) + src_row * row_bytes;
    uint4* dst = reinterpret_cast<uint4*>(a.b_act + slot * (a.K / 2));
    uint8_t* sf_row = a.sfb + sf_offset(e, r, 0, n_rt, n_kt);
    for (int kb0 = lo; kb0 < hi; kb0 += 32) {
      BlockRegs b;
      const int kb = kb0 + lane;
      if (kb < KB) {
        if constexpr (kSrc == kGated) {
          const uint8_t* gate = src + (a.interleaved ? 128LL : 64LL) * kb;
          const uint8_t* up = a.interleaved ? gate + 64 : gate + 64LL * KB;
          BlockRegs g, up_b;
          load_block(gate, wide, g);
          load_block(up, wide, up_b);
          gated_act16(g.lo, up_b.lo, a.act, b.lo);
          gated_act16(g.hi, up_b.hi, a.act, b.hi);
        } else {
          load_block(src + 64LL * kb, wide, b);
          if (weighted) block_weight(b, w);
        }
      }
      finish_blocks(b, kb0, KB, gs, dst, sf_row, lane);
    }
  }
  if (!a.filled) benign_fill_dead<false>(a.counts, a.E, a.cap, n_rt, n_kt, a.sfb);
}

// The same for short rows, rows that leave many lanes of a warp's last 32 K-blocks idle, and destinations that are less
// than 16-byte aligned (pieces of a caller's larger buffer).  The work is the quads of the live rows laid end to end - a
// quad is four K-blocks, one word of scales, four lanes - cut into one range per warp, so that no lane idles whatever the
// row length.  A warp looks up 32 rows at a time, one per lane, and its quads fetch theirs by shuffles: with short rows a
// search per row is a chain of shared-memory reads in front of every few loads.
template <int kSrc>
__global__ void __launch_bounds__(kThreads, kBatchedBlocks)
quant_quads_kernel(const RowsArgs a) {
  extern __shared__ unsigned s_prefix[];
  pdl_wait();
  pdl_launch_dependents();
  const int KB = a.K / kSfBlock;
  const int n_rt = sf_row_atoms(a.cap);
  const int n_kt = sf_k_atoms(a.K);
  const bool wide = (reinterpret_cast<uintptr_t>(a.x) & 31) == 0;
  const bool dst16 = (reinterpret_cast<uintptr_t>(a.b_act) & 15) == 0;
  const int lane = threadIdx.x & 31;
  LiveRows rows;
  rows.make(a.counts, a.E, a.cap, s_prefix);
  const unsigned long long quads = (unsigned long long)rows.total * (unsigned)n_kt;
  const unsigned nwarps = gridDim.x * kWarpsPerBlock;
  const unsigned long long per_warp = (quads + 8ull * nwarps - 1) / (8ull * nwarps) * 8;
  const unsigned long long q0 = per_warp * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x);      // (few ranges: on many SMs)
  if (q0 < quads) {
    int left = (int)min(per_warp, quads - q0) - (lane >> 2);       // quads of the range from this lane's on
    unsigned row0 = (unsigned)(q0 / (unsigned)n_kt);               // first row looked up
    const int kt0 = (int)(q0 - (unsigned long long)row0 * (unsigned)n_kt) + (lane >> 2);
    int b = kt0 / n_kt, kt = kt0 - b * n_kt;                       // this lane's quad: row row0 + b, K-blocks 4 kt ...
    const int step_b = 8 / n_kt, step_kt = 8 - step_b * n_kt;
    const long long row_bytes = (kSrc == kGated ? 4LL : 2LL) * a.K;
    const bool weighted = kSrc == kGather && a.topk_w != nullptr;
    unsigned my_slot = 0;                                          // of row row0 + lane
    int my_e = 0, my_tok = 0;
    float my_w = 1.f;
    bool look = true;
    while (__any_sync(0xffffffffu, left > 0)) {
      if (!look && __any_sync(0xffffffffu, b > 31)) {              // on to the next rows: the first quad's becomes row0
        const int shift = __shfl_sync(0xffffffffu, b, 0);
        row0 += (unsigned)shift;
        b -= shift;
        look = true;
      }
      if (look) {
        look = false;
        const unsigned j = min(row0 + (unsigned)lane, rows.total - 1u);
        int r;
        rows.find_each(j, my_e, r);
        my_slot = my_e < 0 ? 0u : (unsigned)my_e * (unsigned)a.cap + (unsigned)r;
        if constexpr (kSrc == kGather) {
          if (my_e >= 0) {
            my_tok = a.src_tok[my_slot];
            if (weighted) my_w = __bfloat162float(__float2bfloat16_rn(a.topk_w[a.src_route[my_slot]]));
          }
        }
      }
      const int e = __shfl_sync(0xffffffffu, my_e, b);
      const unsigned slot = __shfl_sync(0xffffffffu, my_slot, b);
      long long src_row = slot;
      float w = 1.f;
      if constexpr (kSrc == kGather) {
        src_row = __shfl_sync(0xffffffffu, my_tok, b);
        if (weighted) w = __shfl_sync(0xffffffffu, my_w, b);
      }
      const bool on = left > 0 && e >= 0;
      const int kb = kt * 4 + (lane & 3);
      uint32_t sf_byte = kBenignSf;   // blocks past K keep the benign byte in the layout's slop
      if (on && kb < KB) {
        const float gs = a.gscale[a.gscale_per_expert ? e : 0];
        const uint8_t* src = reinterpret_cast<const uint8_t*>(a.x) + src_row * row_bytes;
        BlockRegs blk;
        if constexpr (kSrc == kGated) {
          const uint8_t* gate = src + (a.interleaved ? 128LL : 64LL) * kb;
          const uint8_t* up = a.interleaved ? gate + 64 : gate + 64LL * KB;
          BlockRegs g, up_b;
          load_block(gate, wide, g);
          load_block(up, wide, up_b);
          gated_act16(g.lo, up_b.lo, a.act, blk.lo);
          gated_act16(g.hi, up_b.hi, a.act, blk.hi);
        } else {
          load_block(src + 64LL * kb, wide, blk);
          if (weighted) block_weight(blk, w);
        }
        float inv;
        block_scale(block_amax(blk), gs, sf_byte, inv);
        store_codes(reinterpret_cast<uint4*>(a.b_act + (long long)slot * (a.K / 2)) + kb, block_codes(blk, inv), dst16);
      }
      const uint32_t word = gather_sf_word(sf_byte);
      if (on && (lane & 3) == 0)
        *reinterpret_cast<uint32_t*>(a.sfb + sf_offset(e, (int)(slot - (unsigned)e * (unsigned)a.cap), kt * 4, n_rt, n_kt)) = word;
      left -= 8;
      b += step_b;
      kt += step_kt;
      if (kt >= n_kt) { kt -= n_kt; ++b; }
    }
  }
  if (!a.filled) benign_fill_dead<true>(a.counts, a.E, a.cap, n_rt, n_kt, a.sfb);
}

// n 16-byte words by one warp, eight of them per lane in flight.
__device__ __forceinline__ void warp_copy(const uint4* __restrict__ src, uint4* __restrict__ dst, int n, int lane) {
  for (int v0 = 0; v0 < n; v0 += 256) {
    uint4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (v0 + i * 32 + lane < n) x[i] = __ldg(src + v0 + i * 32 + lane);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (v0 + i * 32 + lane < n) dst[v0 + i * 32 + lane] = x[i];
  }
}
constexpr int kCopyBlocks = 3;      // blocks per SM of the kernels that copy rows (70 to 80 registers)

// One word of scales: K-blocks 4 kt ... of a row in natural order (`words`: the row can be read by aligned words); blocks
// past K become the benign byte.
__device__ __forceinline__ uint32_t load_sf_word(const uint8_t* sf_src, int kt, int KB, bool words) {
  if (words) return __ldg(reinterpret_cast<const uint32_t*>(sf_src) + kt);
  uint32_t w = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) w |= (kt * 4 + i < KB ? (uint32_t)__ldg(sf_src + kt * 4 + i) : (uint32_t)kBenignSf) << (8 * i);
  return w;
}
// scatter_fp4_planned / scatter_fp4_wire: already quantized rows into the batched operands, one warp per live row.
// Codes are copied 16 bytes per lane; the row's scales go from natural order into the swizzled layout four
// K-blocks (one aligned word of both layouts) at a time.  Slots at or past counts[e] get the benign fill in their scales.
// A warp looks up its next 32 rows at once, one per lane, and copies short rows two or four at a time: the search,
// the source index and the row's first load are a chain of three memory latencies that long rows hide and short ones do not.
// Bound: HBM (65536 rows of 7168: 250 MB in and out in 104 us; a plain fill of 256 MB takes 74).
struct Fp4Rows {
  const uint8_t* q;
  const uint8_t* q_sf;
  uint8_t* b_act;
  uint8_t* sfb;
  long long q_pitch, sf_pitch;
  int K, KB, cap, n_rt, n_kt;
  bool words, dst4;
};
// Rows i0 ... i0 + kRows - 1 of the 32 looked up (slot, token and expert of row i in lane i; expert -1: none).
template <int kRows, int kVecs>                // kVecs: 16-byte words of a row per lane
__device__ __forceinline__ void copy_fp4_rows(const Fp4Rows& a, int i0, int my_e, unsigned my_slot, int my_tok, int lane) {
  const int nv = a.K / 32;
  uint4 x[kRows * kVecs];
  uint32_t sf[kRows];
#pragma unroll
  for (int g = 0; g < kRows; ++g) {
    const bool on = __shfl_sync(0xffffffffu, my_e, i0 + g) >= 0;
    const long long t = __shfl_sync(0xffffffffu, my_tok, i0 + g);
    const uint4* src = reinterpret_cast<const uint4*>(a.q + t * a.q_pitch);
    if (on && lane < a.n_kt) sf[g] = load_sf_word(a.q_sf + t * a.sf_pitch, lane, a.KB, a.words);
#pragma unroll
    for (int c = 0; c < kVecs; ++c)
      if (on && c * 32 + lane < nv) x[g * kVecs + c] = __ldg(src + c * 32 + lane);
  }
#pragma unroll
  for (int g = 0; g < kRows; ++g) {
    const int e = __shfl_sync(0xffffffffu, my_e, i0 + g);
    const unsigned slot = __shfl_sync(0xffffffffu, my_slot, i0 + g);
    if (e < 0) continue;
    uint4* dst = reinterpret_cast<uint4*>(a.b_act + (long long)slot * (a.K / 2));
    if (lane < a.n_kt)
      store_sf_word(a.sfb + sf_offset(e, (int)(slot - (unsigned)e * (unsigned)a.cap), lane * 4, a.n_rt, a.n_kt), sf[g], a.dst4);
#pragma unroll
    for (int c = 0; c < kVecs; ++c)
      if (c * 32 + lane < nv) dst[c * 32 + lane] = x[g * kVecs + c];
  }
}
// kRows: rows a warp copies at a time, each of at most 32 * kVecs 16-byte words; 1: long rows, one after the other.
template <int kRows, int kVecs>
__global__ void __launch_bounds__(kThreads, kCopyBlocks)
scatter_fp4_rows_kernel(const uint8_t* __restrict__ q, long long q_pitch, const uint8_t* __restrict__ q_sf,
                        long long sf_pitch, const int* __restrict__ src_tok, const int* __restrict__ counts, int K, int E,
                        int cap, uint8_t* __restrict__ b_act, uint8_t* __restrict__ sfb, int filled) {
  extern __shared__ unsigned s_prefix[];
  pdl_wait();
  pdl_launch_dependents();
  const int KB = K / kSfBlock;
  const bool words = (KB % 4) == 0 && (sf_pitch % 4) == 0 && (reinterpret_cast<uintptr_t>(q_sf) % 4) == 0;
  const Fp4Rows a{q, q_sf, b_act, sfb, q_pitch, sf_pitch, K, KB, cap, sf_row_atoms(cap), sf_k_atoms(K), words,
                  (reinterpret_cast<uintptr_t>(sfb) % 4) == 0};
  const int lane = threadIdx.x & 31;
  LiveRows rows;
  rows.make(counts, E, cap, s_prefix);
  const unsigned nwarps = gridDim.x * kWarpsPerBlock;
  for (unsigned j0 = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); j0 < rows.total; j0 += 32u * nwarps) {
    const unsigned long long j = j0 + (unsigned long long)lane * nwarps;  // this lane looks up the warp's row number `lane`
    const bool there = j < rows.total;
    int e, r, tok = 0;
    rows.find_each(there ? (unsigned)j : j0, e, r);
    if (!there) e = -1;
    const unsigned slot = e < 0 ? 0u : (unsigned)e * (unsigned)cap + (unsigned)r;
    if (e >= 0) tok = src_tok[slot];
    const int n = (int)min(32u, (rows.total - j0 + nwarps - 1) / nwarps);
    if constexpr (kRows > 1) {
#pragma unroll 1
      for (int i = 0; i < n; i += kRows) copy_fp4_rows<kRows, kVecs>(a, i, e, slot, tok, lane);
    } else {
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        const int ei = __shfl_sync(0xffffffffu, e, i);
        const unsigned si = __shfl_sync(0xffffffffu, slot, i);
        const long long t = __shfl_sync(0xffffffffu, tok, i);
        if (ei < 0) continue;
        uint8_t* sf_row = sfb + sf_offset(ei, (int)(si - (unsigned)ei * (unsigned)cap), 0, a.n_rt, a.n_kt);
#pragma unroll 1
        for (int kt = lane; kt < a.n_kt; kt += 32)
          store_sf_word(sf_row + kt * 512, load_sf_word(q_sf + t * sf_pitch, kt, KB, words), a.dst4);
        warp_copy(reinterpret_cast<const uint4*>(q + t * q_pitch), reinterpret_cast<uint4*>(b_act + (long long)si * (K / 2)), K / 32, lane);
      }
    }
  }
  if (!filled) benign_fill_dead_atoms(counts, E, cap, a.n_rt, a.n_kt, sfb);
}

// quant_rows: token-order rows -> row-major codes and natural-order scales, one shared global scale.
// One warp per row, one 32-element block per lane; four scales leave as one word.
__global__ void __launch_bounds__(kThreads)
quant_rows_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gscale, unsigned T, int K,
                  uint8_t* __restrict__ q, uint8_t* __restrict__ q_sf) {
  pdl_wait();
  pdl_launch_dependents();
  const int KB = K / kSfBlock;
  const int lane = threadIdx.x & 31;
  const float gs = gscale[0];
  const unsigned warp0 = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  const unsigned nwarps = gridDim.x * kWarpsPerBlock;
  const bool sf_words = (KB % 4) == 0;     // rows of scales are then 4-byte aligned
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 31) == 0;
  for (unsigned t = warp0; t < T; t += nwarps) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(x + (long long)t * K);
    uint4* dst = reinterpret_cast<uint4*>(q + (long long)t * (K / 2));
    uint8_t* sf_row = q_sf + (long long)t * KB;
    for (int kb0 = 0; kb0 < KB; kb0 += 32) {
      const int kb = kb0 + lane;
      uint32_t sf_byte = 0;
      if (kb < KB) {
        BlockRegs b;
        load_block(src + 64LL * kb, wide, b);
        float inv;
        block_scale(block_amax(b), gs, sf_byte, inv);
        dst[kb] = block_codes(b, inv);
        if (!sf_words) sf_row[kb] = (uint8_t)sf_byte;
      }
      const uint32_t word = gather_sf_word(sf_byte);
      if (sf_words && (lane & 3) == 0 && kb < KB) *reinterpret_cast<uint32_t*>(sf_row + kb) = word;
    }
  }
}

// The activation alone, 16 features (32 bytes of gate, up and result) per thread.  Bound: HBM (131072 rows of 2 x 2048).
__global__ void __launch_bounds__(kThreads)
gated_act_kernel(const __nv_bfloat16* __restrict__ x2, long long rows, int N, int interleaved,
                 GatedAct act, __nv_bfloat16* __restrict__ y) {
  const int per_row = N / 16;
  const long long total = rows * per_row;
  const bool wide = (reinterpret_cast<uintptr_t>(x2) & 31) == 0;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long row = idx / per_row;
    const int k0 = (int)(idx - row * per_row) * 16;
    const __nv_bfloat16* base = x2 + row * (2LL * N);
    const int gate_off = interleaved ? (k0 / 32) * 64 + (k0 % 32) : k0;
    const int up_off = interleaved ? gate_off + 32 : N + k0;
    uint32_t g[8], u[8], o[8];
    load32(reinterpret_cast<const uint8_t*>(base + gate_off), wide, g);
    load32(reinterpret_cast<const uint8_t*>(base + up_off), wide, u);
    gated_act16(g, u, act, o);
    uint4* dst = reinterpret_cast<uint4*>(y + row * N + k0);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

// Wire rows of the expert-parallel dispatch: one routed token row as it crosses the link,
//   [K/2 bytes of e2m1 codes][K/32 UE4M3 scales][padding to 16 bytes][int32 expert id local to the receiver][12 bytes]
// in fixed-capacity slabs of `slab` rows per destination rank.  Slot s of slab w is live when
// s < slab_counts[w]; a dead slot only gets its expert id, -1, which the receiver's dispatch_plan
// treats like any routing that is not for one of its experts.
__host__ __device__ inline long long wire_row_bytes(int K) { return (long long)round_up_i(K / 2 + K / kSfBlock, 16) + 16; }

// One warp per slot, all of a row's words in flight at once.  Bound: writes to HBM (65536 rows of 3840 bytes: 75 us, as a
// plain fill of as many bytes; with a block of 128 threads per slot and its three dependent loads 85).
template <class IdT>
__global__ void __launch_bounds__(kThreads)
pack_wire_rows_kernel(const uint8_t* __restrict__ q, const uint8_t* __restrict__ q_sf, const IdT* __restrict__ ids,
                      const int* __restrict__ slot_tok, const int* __restrict__ slot_route,
                      const int* __restrict__ slab_counts, unsigned slots, int slab, int experts_per_rank, int K,
                      uint8_t* __restrict__ wire, const RowParts parts) {
  pdl_wait();
  pdl_launch_dependents();
  const long long row_bytes = wire_row_bytes(K);
  const int KB = K / kSfBlock;
  const int lane = threadIdx.x & 31;
  const unsigned nwarps = gridDim.x * kWarpsPerBlock;
  for (unsigned slot = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); slot < slots; slot += nwarps) {
    const int w = (int)(slot / (unsigned)slab);
    const int s = (int)(slot - (unsigned)w * (unsigned)slab);
    // (with parts: slab w goes to buffer w, which may be the receiving rank's own memory)
    uint8_t* row = parts.n ? static_cast<uint8_t*>(parts.base[w]) + s * row_bytes : wire + slot * row_bytes;
    int* id_out = reinterpret_cast<int*>(row + row_bytes - 16);
    if (s >= min(slab_counts[w], slab)) {
      if (lane == 0) *id_out = -1;
      continue;
    }
    const long long t = slot_tok[slot];
    const int route = slot_route[slot];
    const uint8_t* sf_src = q_sf + t * KB;
    uint8_t* sf_dst = row + K / 2;
    if (KB % 16 == 0) {
      for (int v = lane; v < KB / 16; v += 32)
        reinterpret_cast<uint4*>(sf_dst)[v] = __ldg(reinterpret_cast<const uint4*>(sf_src) + v);
    } else {
      for (int b = lane; b < KB; b += 32) sf_dst[b] = __ldg(sf_src + b);
    }
    warp_copy(reinterpret_cast<const uint4*>(q + t * (K / 2)), reinterpret_cast<uint4*>(row), K / 32, lane);
    if (lane == 0) *id_out = (int)((long long)ids[route] - (long long)w * experts_per_rank);
  }
}

int grid_for(long long warp_items, int sm_count, int per_sm = 8) {      // 8 x 256 threads fill an SM
  long long blocks = (warp_items + kWarpsPerBlock - 1) / kWarpsPerBlock;
  long long cap = (long long)(sm_count > 0 ? sm_count : 148) * per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

bool aligned_to(const void* p, unsigned n) { return reinterpret_cast<uintptr_t>(p) % n == 0; }

// What the row kernels' vector accesses need of their pointers (a bf16 source is read 16 bytes at a time).
int check_alignment(const void* x, const uint8_t* b_act, unsigned b_align, const uint8_t* sfb) {
  PNV_REQUIRE(aligned_to(x, 16), "the bf16 source must be 16-byte aligned");
  PNV_REQUIRE(aligned_to(b_act, b_align), "the codes must be %u-byte aligned", b_align);
  PNV_REQUIRE(aligned_to(sfb, 4), "the scales must be 4-byte aligned");
  return PNV_OK;
}

int check_common(const void* x, const float* gscale, const int32_t* counts, int E, int rows, int K,
                 const uint8_t* b_act, const uint8_t* sfb, const char* kname) {
  PNV_REQUIRE(x && gscale && counts && b_act && sfb, "null pointer argument");
  PNV_REQUIRE(E >= 1 && rows >= 1, "experts and row capacity must be positive, got %d and %d", E, rows);
  PNV_REQUIRE(K > 0 && K % kSfBlock == 0, "%s must be a multiple of %d, got %d", kname, kSfBlock, K);
  PNV_REQUIRE(sf_numel(rows, K, E) / 16 < (1LL << 31) - (1LL << 24), "the scale layout has too many lines for one launch");
  PNV_REQUIRE(sf_numel(rows, K, E) / 16 < (1LL << 40), "scale buffer too large");
  return PNV_OK;
}

// The planned scatters' fill.  Rows between the capacity and the end of its last 128-row atom are dead whatever the counts
// say.  Where they are many - thousands of experts of a few rows - the whole scale buffer is filled by a memset first, which
// writes faster than the row kernels' own fill; otherwise the row kernels do it and can start while their predecessor
// drains.  The lines, measured: rows copied for 2048 experts x 16 x 7168 (49 MiB surely dead) 58 us with a memset, 62
// without, below that the memset loses; rows quantized for 2048 experts 92 us with, 85 without, for 9000 x 4 x 7168
// (238 MiB) 137 with, 160 without.
constexpr long long kMemsetFillCopy = 40LL << 20, kMemsetFillQuant = 96LL << 20;
int fill_ahead(uint8_t* sfb, int E, int cap, int K, long long least, cudaStream_t s, int& filled) {
  const long long surely_dead = (long long)E * ((long long)sf_row_atoms(cap) * 128 - cap) * sf_k_atoms(K) * 4;
  filled = surely_dead >= least ? 1 : 0;
  if (filled) PNV_CUDA(cudaMemsetAsync(sfb, kBenignSf, (size_t)sf_numel(cap, K, E), s));
  return PNV_OK;
}

// One launch of the shared kernel: at most a wave of warps, one per 32 K-blocks of a row of the capacity (or eight quads).
template <int kSrc>
int launch_batched(RowsArgs a, int sm_count, cudaStream_t s) {
  if (int rc = check_alignment(a.x, a.b_act, kSrc == kGather ? 16 : 8, a.sfb)) return rc;
  if (kSrc == kGather) PNV_REQUIRE((long long)a.E * a.cap < (1LL << 31), "E * cap must fit int32");
  // (a grid stride short of 2^32, so that a warp's next row number cannot wrap around)
  PNV_REQUIRE((long long)a.E * a.cap < (1LL << 32) - (1LL << 24), "experts * max_n must be below 2^32 - 2^24");
  if (kSrc == kGather)
    if (int rc = fill_ahead(a.sfb, a.E, a.cap, a.K, kMemsetFillQuant, s, a.filled)) return rc;
  const int KB = a.K / kSfBlock;
  // A warp per row where rows are long (64 K-blocks) and at most a sixteenth of its lanes would idle: the row's addresses
  // and its lookup then serve many blocks.  Also where the whole capacity is no more than one step for each warp of a wave:
  // idle lanes then cost nothing, and the row form starts sooner (the grouped linear layer of 5 experts x 1 row x 4608: 13.0
  // us against 13.3).
  const long long steps = (long long)a.E * a.cap * ceil_div_i(KB, 32);
  const long long wave = (long long)(sm_count > 0 ? sm_count : 148) * kBatchedBlocks * kWarpsPerBlock;
  const bool rows = aligned_to(a.b_act, 16) && aligned_to(a.sfb, 16) &&
                    (steps <= wave || (KB >= 64 && 16 * (round_up_i(KB, 32) - KB) <= KB));
  const long long units = rows ? steps : ((long long)a.E * a.cap * sf_k_atoms(a.K) + 7) / 8;
  PNV_CUDA(launch_pdl(rows ? quant_batched_kernel<kSrc> : quant_quads_kernel<kSrc>,
                      dim3(grid_for(units, sm_count, kBatchedBlocks)), dim3(kThreads), live_rows_smem(a.E), s, pdl_enabled() && !a.filled, a));
  return PNV_OK;
}

}  // namespace

static bool g_silu_short = true;

int make_gated_act(int act_kind, float beta, float linear_beta, GatedAct& out) {
  if (act_kind == PNV_ACT_SILU) {
    out = GatedAct{PNV_ACT_SILU, 1.0f, -1.0f, 1.0f, -1.0f, g_silu_short ? 0 : 1};
  } else if (act_kind == PNV_ACT_SITU) {
    PNV_REQUIRE(beta > 0, "situ: beta must be positive, got %g", (double)beta);
    out = GatedAct{PNV_ACT_SITU, beta, linear_beta, 1.0f / beta, 1.0f / linear_beta, 0};
  } else {
    return fail(PNV_ERR_INVALID_ARGUMENT, "activation must be 'silu' or 'situ', got kind %d", act_kind);
  }
  return PNV_OK;
}

}  // namespace pnv

using namespace pnv;

extern "C" int pnv_quant_act(const void* x, const float* gscale, int gscale_per_expert,
                             const int32_t* counts, int experts, int max_n, int k, uint8_t* b_act,
                             uint8_t* sfb, int sm_count, pnv_stream_t stream) {
  if (int rc = check_common(x, gscale, counts, experts, max_n, k, b_act, sfb, "K")) return rc;
  RowsArgs a{(const __nv_bfloat16*)x, nullptr, nullptr, nullptr, gscale, (const int*)counts, b_act, sfb, GatedAct{},
             gscale_per_expert, experts, max_n, k, 0, 0};
  return launch_batched<kPlain>(a, sm_count, (cudaStream_t)stream);
}

extern "C" int pnv_silu_mul_quant_act(const void* x2, const float* gscale, int gscale_per_expert,
                                      const int32_t* counts, int experts, int max_n, int n,
                                      int interleaved, int act_kind, float beta, float linear_beta,
                                      uint8_t* b_act, uint8_t* sfb, int sm_count,
                                      pnv_stream_t stream) {
  GatedAct act;
  if (int rc = make_gated_act(act_kind, beta, linear_beta, act)) return rc;
  if (int rc = check_common(x2, gscale, counts, experts, max_n, n, b_act, sfb, "intermediate width N"))
    return rc;
  RowsArgs a{(const __nv_bfloat16*)x2, nullptr, nullptr, nullptr, gscale, (const int*)counts, b_act, sfb, act,
             gscale_per_expert, experts, max_n, n, interleaved ? 1 : 0, 0};
  return launch_batched<kGated>(a, sm_count, (cudaStream_t)stream);
}

extern "C" int pnv_scatter_quant_act(const void* a1, const int64_t* flat_tok,
                                     const int64_t* dest_global, const float* topk_weights,
                                     const float* gscale, int gscale_per_expert, int64_t n_routes,
                                     int k, int experts, int cap, uint8_t* b_act, uint8_t* sfb,
                                     int sm_count, pnv_stream_t stream) {
  PNV_REQUIRE(cap > 0, "cap must be positive");
  PNV_REQUIRE(n_routes >= 0, "n_routes must be non-negative");
  PNV_REQUIRE(n_routes == 0 || (flat_tok && dest_global), "null routing plan");
  int dummy = 0;
  if (int rc = check_common(a1 ? a1 : (const void*)&dummy, gscale, &dummy, experts, cap, k, b_act, sfb, "K"))
    return rc;
  PNV_REQUIRE(n_routes == 0 || a1, "null pointer argument");
  if (n_routes > 0)
    if (int rc = check_alignment(a1, b_act, 16, sfb)) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  PNV_CUDA(cudaMemsetAsync(sfb, kBenignSf, (size_t)sf_numel(cap, k, experts), s));
  if (n_routes == 0) return PNV_OK;
  PNV_REQUIRE(n_routes < (1LL << 31) && (long long)experts * cap < (1LL << 31), "T * topk and E * cap must fit int32");
  PNV_CUDA(launch_pdl(scatter_quant_kernel, dim3(grid_for(n_routes, sm_count)), dim3(kThreads), 0, s,
                      false, (const __nv_bfloat16*)a1, (const long long*)flat_tok,
                      (const long long*)dest_global, topk_weights, gscale, gscale_per_expert,
                      (unsigned)n_routes, k, experts, cap, b_act, sfb));
  return PNV_OK;
}

extern "C" int pnv_gated_act(const void* x2, int64_t rows, int n, int interleaved, int act_kind,
                             float beta, float linear_beta, void* y, pnv_stream_t stream) {
  GatedAct act;
  if (int rc = make_gated_act(act_kind, beta, linear_beta, act)) return rc;
  PNV_REQUIRE(x2 && y, "null pointer argument");
  PNV_REQUIRE(n > 0 && n % kSfBlock == 0, "intermediate width N must be a multiple of %d, got %d", kSfBlock, n);
  if (rows <= 0) return PNV_OK;
  PNV_REQUIRE(aligned_to(x2, 16) && aligned_to(y, 16), "gated_act buffers must be 16-byte aligned");
  long long total = rows * (n / 16);
  long long blocks = (total + kThreads - 1) / kThreads;
  if (blocks > 148LL * 32) blocks = 148LL * 32;
  gated_act_kernel<<<(unsigned)blocks, kThreads, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x2, (long long)rows, n, interleaved ? 1 : 0, act, (__nv_bfloat16*)y);
  PNV_CUDA(cudaGetLastError());
  return PNV_OK;
}

extern "C" int pnv_scatter_quant_act_planned(const void* a1, const int32_t* src_tok, const int32_t* src_route,
                                             const float* topk_weights, const float* gscale, int gscale_per_expert,
                                             const int32_t* counts, int k, int experts, int cap, uint8_t* b_act,
                                             uint8_t* sfb, int sm_count, pnv_stream_t stream) {
  PNV_REQUIRE(cap > 0, "cap must be positive");
  PNV_REQUIRE(src_tok && src_route, "null pointer argument");
  if (int rc = check_common(a1, gscale, counts, experts, cap, k, b_act, sfb, "K")) return rc;
  RowsArgs a{(const __nv_bfloat16*)a1, (const int*)src_tok, (const int*)src_route, topk_weights, gscale, (const int*)counts,
             b_act, sfb, GatedAct{}, gscale_per_expert, experts, cap, k, 0, 0};
  return launch_batched<kGather>(a, sm_count, (cudaStream_t)stream);
}

extern "C" int pnv_quant_rows(const void* x, const float* gscale, int64_t tokens, int k, uint8_t* q, uint8_t* q_sf,
                              int sm_count, pnv_stream_t stream) {
  PNV_REQUIRE(k > 0 && k % kSfBlock == 0, "K must be a multiple of %d, got %d", kSfBlock, k);
  PNV_REQUIRE(tokens >= 0, "bad token count");
  if (tokens == 0) return PNV_OK;
  PNV_REQUIRE(x && gscale && q && q_sf, "null pointer argument");
  PNV_REQUIRE(tokens < (1LL << 31), "too many tokens");
  PNV_REQUIRE(aligned_to(x, 16) && aligned_to(q, 16), "quant_rows: the bf16 rows and the codes must be 16-byte aligned");
  PNV_REQUIRE((k / kSfBlock) % 4 != 0 || aligned_to(q_sf, 4), "quant_rows: the scales must be 4-byte aligned");
  PNV_CUDA(launch_pdl(quant_rows_kernel, dim3(grid_for(tokens, sm_count)), dim3(kThreads), 0, (cudaStream_t)stream,
                      pdl_enabled(), (const __nv_bfloat16*)x, gscale, (unsigned)tokens, k, q, q_sf));
  return PNV_OK;
}

namespace {
int scatter_fp4_rows(const uint8_t* q, long long q_pitch, const uint8_t* q_sf, long long sf_pitch, const int32_t* src_tok,
                     const int32_t* counts, int k, int experts, int cap, uint8_t* b_act, uint8_t* sfb, int sm_count,
                     cudaStream_t s) {
  float dummy = 0.f;
  if (int rc = check_common(q, &dummy, counts, experts, cap, k, b_act, sfb, "K")) return rc;
  PNV_REQUIRE((long long)experts * cap < (1LL << 31), "E * cap must fit int32");
  PNV_REQUIRE((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(b_act) | (uintptr_t)q_pitch) % 16 == 0,
              "code rows must be 16-byte aligned");
  int filled = 0;
  if (int rc = fill_ahead(sfb, experts, cap, k, kMemsetFillCopy, s, filled)) return rc;
  const int nv = k / 32;
  auto kernel = nv <= 32 ? scatter_fp4_rows_kernel<4, 1> : nv <= 64 ? scatter_fp4_rows_kernel<4, 2>
              : nv <= 128 ? scatter_fp4_rows_kernel<2, 4> : scatter_fp4_rows_kernel<1, 8>;
  PNV_CUDA(launch_pdl(kernel, dim3(grid_for((long long)experts * cap, sm_count, kCopyBlocks)), dim3(kThreads),
                      live_rows_smem(experts), s, pdl_enabled() && !filled, q, q_pitch, q_sf, sf_pitch, (const int*)src_tok,
                      (const int*)counts, k, experts, cap, b_act, sfb, filled));
  return PNV_OK;
}
}  // namespace

extern "C" int pnv_scatter_fp4_planned(const uint8_t* q, const uint8_t* q_sf, const int32_t* src_tok,
                                       const int32_t* counts, int k, int experts, int cap, uint8_t* b_act,
                                       uint8_t* sfb, int sm_count, pnv_stream_t stream) {
  PNV_REQUIRE(cap > 0, "cap must be positive");
  PNV_REQUIRE(q && q_sf && src_tok, "null pointer argument");
  PNV_REQUIRE(k > 0 && k % kSfBlock == 0, "K must be a multiple of %d, got %d", kSfBlock, k);
  return scatter_fp4_rows(q, k / 2, q_sf, k / kSfBlock, src_tok, counts, k, experts, cap, b_act, sfb, sm_count,
                          (cudaStream_t)stream);
}

extern "C" int pnv_set_silu_table(int enabled) {
  g_silu_short = enabled != 0;
  return PNV_OK;
}


extern "C" int64_t pnv_wire_row_bytes(int k) {
  if (k <= 0 || k % kSfBlock != 0) return 0;
  return wire_row_bytes(k);
}

namespace {
int pack_wire_rows_common(const uint8_t* q, const uint8_t* q_sf, const void* topk_ids, int ids_are_int64,
                          const int32_t* slot_tok, const int32_t* slot_route, const int32_t* slab_counts, int ranks,
                          int slab, int experts_per_rank, int k, uint8_t* wire, const RowParts& parts,
                          pnv_stream_t stream) {
  PNV_REQUIRE(k > 0 && k % kSfBlock == 0, "K must be a multiple of %d, got %d", kSfBlock, k);
  PNV_REQUIRE(ranks >= 1 && slab >= 1 && experts_per_rank >= 1, "ranks, slab and experts_per_rank must be positive");
  PNV_REQUIRE((long long)ranks * slab < (1LL << 31), "ranks * slab must fit int32");
  PNV_REQUIRE(q && q_sf && topk_ids && slot_tok && slot_route && slab_counts, "null pointer argument");
  PNV_REQUIRE((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(wire)) % 16 == 0 &&
                  ((k / kSfBlock) % 16 != 0 || reinterpret_cast<uintptr_t>(q_sf) % 16 == 0),
              "pack_wire_rows buffers must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned slots = (unsigned)(ranks * slab);
  const dim3 grid((unsigned)grid_for(slots, 0, kCopyBlocks)), block(kThreads);
  if (ids_are_int64)
    PNV_CUDA(launch_pdl(pack_wire_rows_kernel<long long>, grid, block, 0, s, pdl_enabled(), q, q_sf,
                        (const long long*)topk_ids, (const int*)slot_tok, (const int*)slot_route,
                        (const int*)slab_counts, slots, slab, experts_per_rank, k, wire, parts));
  else
    PNV_CUDA(launch_pdl(pack_wire_rows_kernel<int>, grid, block, 0, s, pdl_enabled(), q, q_sf, (const int*)topk_ids,
                        (const int*)slot_tok, (const int*)slot_route, (const int*)slab_counts, slots, slab,
                        experts_per_rank, k, wire, parts));
  return PNV_OK;
}
}  // namespace

extern "C" int pnv_pack_wire_rows(const uint8_t* q, const uint8_t* q_sf, const void* topk_ids, int ids_are_int64,
                                  const int32_t* slot_tok, const int32_t* slot_route, const int32_t* slab_counts,
                                  int ranks, int slab, int experts_per_rank, int k, uint8_t* wire,
                                  pnv_stream_t stream) {
  PNV_REQUIRE(wire, "null pointer argument");
  RowParts none{};
  return pack_wire_rows_common(q, q_sf, topk_ids, ids_are_int64, slot_tok, slot_route, slab_counts, ranks, slab,
                               experts_per_rank, k, wire, none, stream);
}

extern "C" int pnv_pack_wire_rows_parts(const uint8_t* q, const uint8_t* q_sf, const void* topk_ids, int ids_are_int64,
                                        const int32_t* slot_tok, const int32_t* slot_route,
                                        const int32_t* slab_counts, int ranks, int slab, int experts_per_rank, int k,
                                        void* const* wire_parts, pnv_stream_t stream) {
  RowParts parts;
  if (int rc = make_row_parts(wire_parts, ranks, slab, parts)) return rc;
  return pack_wire_rows_common(q, q_sf, topk_ids, ids_are_int64, slot_tok, slot_route, slab_counts, ranks, slab,
                               experts_per_rank, k, nullptr, parts, stream);
}

extern "C" int pnv_scatter_fp4_wire(const uint8_t* wire, const int32_t* src_tok, const int32_t* counts, int k,
                                    int experts, int cap, uint8_t* b_act, uint8_t* sfb, int sm_count,
                                    pnv_stream_t stream) {
  PNV_REQUIRE(cap > 0, "cap must be positive");
  PNV_REQUIRE(wire && src_tok, "null pointer argument");
  PNV_REQUIRE(k > 0 && k % kSfBlock == 0, "K must be a multiple of %d, got %d", kSfBlock, k);
  const long long pitch = wire_row_bytes(k);
  return scatter_fp4_rows(wire, pitch, wire + k / 2, pitch, src_tok, counts, k, experts, cap, b_act, sfb, sm_count,
                          (cudaStream_t)stream);
}
