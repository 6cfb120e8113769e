// group_mm, wide token tiles (64 to 256 tokens per tile): prefill-sized problems.
//
// Included by group_mm.cu inside namespace pnv::{anonymous}, after Params and the status codes.
//
// One kernel in two forms.
//   single CTA (kPair = false)  one CTA per SM multiplies 128 weight rows by TILE_N tokens per tile.
//   CTA pair   (kPair = true)   a cluster of two CTAs on neighbouring SMs multiplies 256 weight rows by
//                               TILE_N tokens with one tcgen05.mma.sp.cta_group::2 per 128-K block.  Each
//                               CTA loads its own 128 weight rows (with their metadata and scales) and HALF
//                               of the token rows into its own shared memory with ordinary TMA copies (no
//                               cluster multicast anywhere), and the tensor cores of both SMs read the two
//                               halves.  Against the single-CTA form that halves the activation bytes an SM
//                               has to pull from L2 per unit of math, which is what bounds these shapes.  Both
//                               CTAs' tile loads count their bytes on the first CTA's barrier (.cta_group::2
//                               tiled loads), the second CTA's small bulk copies are relayed by a remote arrive.
//
// Tail tiles.  The last token tile of an expert is often nearly empty (256 +- 16 rows per expert leave every other
// expert a second tile of a dozen rows).  When it holds at most 64 live rows - and the launch has the tensor map for
// it (K a multiple of 256, tiles of 128 tokens or more) - the tile runs 64 tokens wide: a quarter or half of the
// activation bytes, one scale row-atom, MMAs a quarter or half as long.  Every role derives the width from counts[].
// The pair kernel with 256-token tiles has a variant (kDblTails) that multiplies such a tile against two M units per
// work item (WideCfg::kTailDouble); the host picks it when experts hold few token tiles.
//
// 20 warps per CTA.  The first four are single-warp roles whose 32 lanes all follow the role's loop while one elected
// lane issues: TMA, bulk-copy and tcgen05 instructions take their operands from uniform registers, and issued by a lane
// that a thread-index test picked each cost 85 cycles and more of set-up (an elected one 20-60).  That alone took the
// fused gate_up GEMM of 32 experts x 2048 rows x 7168 from 753 to 621 us and one of 8 experts x 25 rows from 98 to 64 us.
//   warp 0   tile producer: TMA copies of the compressed weights and of the activations
//   warp 1   side producer: bulk copies of the metadata, SFA and SFB atoms (they sit in global memory in
//            the shape tensor memory wants)
//   warp 2   MMA issuer (of a pair: in the first CTA only): per pipeline stage one wait, the MMAs and a commit;
//            consecutive tiles go to alternate accumulators where there are two
//   warp 3   copier (of a pair: in the first CTA only): tcgen05.cp of every stage's scale and metadata atoms from
//            shared memory into the stage's slot of a ring in tensor memory, then a tcgen05.commit that tells the issuer
//            the slot is filled.  In the second CTA of a pair it only relays "my side copies have landed".
//   4 - 19   epilogue, four groups of four warps (one warp per lane quarter); a tile's chunks of token
//            columns are dealt round-robin to the groups
// 20 warps leave 96 registers a thread (five warps to each quarter of the SM); 21 or more leave 80, which spilled much more:
// at 96 the plain 256-token forms spill 12 to 24 bytes a thread, the others nothing.
//
// Barriers per pipeline stage s: full[s] (this CTA's copies landed; in a pair's first CTA it also counts the
// second CTA's tile loads), peer_full[s] (pair: the second CTA's bulk copies landed, relayed to the first), sf_full[s]
// (copier's commit -> issuer: scales and metadata are in tensor memory), empty[s] (issuer's tcgen05.commit, delivered
// to both CTAs of a pair -> producers).  Per accumulator stage: acc_full (commit, both CTAs), acc_empty (all epilogue
// warps of the CTA or pair -> issuer).  Every wait is bounded.
//
// What bounds it.  A CTA's TMA takes in about 64 bytes per cycle when its requests are 128 bytes wide; a 64-byte
// request costs as much as a 128-byte one.  Hence 512-K stages (128-byte weight rows) in the 256 x 256 pair wherever K has more
// than 256 (the other variants run the stage depth of their names):
// 953 cycles per 58 KB stage of the 256 x 256 pair without an epilogue, against 815 per 29 KB with 256-K stages.  Short
// K loops are bound by the epilogue instead (see there).

template <int TILE_N, int STAGE_K, bool kPair, bool kDblTails = false>
struct WideCfg {
  static_assert(TILE_N == 64 || TILE_N == 128 || TILE_N == 256, "wide tile widths: 64, 128, 256");
  static_assert(STAGE_K == 256 || STAGE_K == 512, "stage depths: 256, 512");
  static constexpr int kCtas = kPair ? 2 : 1;
  static constexpr int kEpilogueWarps = 16;
  static constexpr int kFirstEpilogueWarp = 4;
  static constexpr int kThreads = (kFirstEpilogueWarp + kEpilogueWarps) * 32;
  static constexpr int kAtoms = STAGE_K / 128;
  static constexpr int kARowBytes = STAGE_K / 4;
  static constexpr int kABytes = kTileM * kARowBytes;
  static constexpr uint32_t kASwizzle = STAGE_K == 512 ? 2 : 4;
  static constexpr int kBRows = TILE_N / kCtas;              // token rows this CTA loads
  static constexpr int kBBoxes = STAGE_K / 256;
  static constexpr int kBBoxBytes = kBRows * 128;
  static constexpr int kBBytes = kBBoxes * kBBoxBytes;
  static constexpr int kEAtoms = STAGE_K / 256;
  static constexpr int kEBytes = 2048 * kEAtoms;
  static constexpr int kSfaBytes = 512 * kAtoms;
  static constexpr int kSfbRowAtoms = TILE_N > 128 ? 2 : 1;  // every CTA holds the scales of all TILE_N tokens
  static constexpr int kSfbBytes = kSfaBytes * kSfbRowAtoms;
  // a pipeline stage in shared memory: [weights | activations | metadata | weight scales | activation scales]
  static constexpr int kStageBytes = kABytes + kBBytes + kEBytes + kSfaBytes + kSfbBytes;
  static constexpr int kOffA = 0;
  static constexpr int kOffB = kABytes;
  static constexpr int kOffE = kOffB + kBBytes;
  static constexpr int kOffSfa = kOffE + kEBytes;
  static constexpr int kOffSfb = kOffSfa + kSfaBytes;
  static constexpr int kTailN = 64;                          // width of a narrow tail tile
  static constexpr int kTailBRows = kTailN / kCtas;
  static constexpr int kTailBBoxBytes = kTailBRows * 128;
  static constexpr int kChunk = TILE_N >= 128 ? 32 : 16;     // token columns an epilogue group takes at a time
  static constexpr int kOutBytes = 4 * 8192;                 // epilogue: one 8 KiB staging area per group
  static constexpr int kBarrierBytes = 1024;
  static constexpr int kMaxStages = 12;
  static constexpr int kAccStages = TILE_N == 256 ? 1 : 2;
  // tensor-memory columns: accumulators below 256, then a ring of slots, one per pipeline stage, each holding
  // the stage's weight scales, activation scales and metadata
  static constexpr int kColSlots = 256;
  static constexpr int kSfbColsPerAtom = 4 * kSfbRowAtoms;
  static constexpr int kSlotSfb = 4 * kAtoms;                // column offsets inside a slot
  static constexpr int kSlotE = kSlotSfb + kSfbColsPerAtom * kAtoms;
  // Double tail items (CTA pairs, 256-token tiles).  A narrow tail tile costs a pipeline stage per
  // 256 K like any other tile although it moves half the bytes and a quarter of the math, so such a tile is
  // multiplied against TWO M units per work item: the stage then holds both units' weights, metadata and weight
  // scales next to the one 64-token activation box, and the item writes two 64-column accumulators.  Half as many
  // stages per tail tile, and the activation box is fetched once for two units.  The support costs every item a few
  // instructions in roles whose instruction streams bound the pipeline, so it is a kernel variant of its own
  // (kDblTails), which the host picks when experts hold few token tiles.  The layout of such a stage:
  static constexpr bool kTailDouble = kDblTails && kPair && TILE_N == 256;
  static constexpr int kDblOffA1 = kABytes;                              // second unit's weights
  static constexpr int kDblOffB = 2 * kABytes;
  static constexpr int kDblOffE = kDblOffB + kBBoxes * kTailBBoxBytes;   // metadata, unit after unit
  static constexpr int kDblOffSfa = kDblOffE + 2 * kEBytes;              // weight scales, unit after unit
  static constexpr int kDblOffSfb = kDblOffSfa + 2 * kSfaBytes;          // activation scales (one row atom)
  static constexpr int kDblBytes = kDblOffSfb + kSfaBytes;
  // ... and of its tensor-memory slot: [SFA unit 0 | SFA unit 1 | SFB | E unit 0 | E unit 1]
  static constexpr int kDblSlotSfa1 = 4 * kAtoms;
  static constexpr int kDblSlotSfb = 8 * kAtoms;
  static constexpr int kDblSlotE = kDblSlotSfb + 4 * kAtoms;
  static constexpr int kDblSlotE1 = kDblSlotE + 4 * kEAtoms;
  static constexpr int kDblSlotCols = kDblSlotE1 + 4 * kEAtoms;
  static constexpr int kSlotCols = kTailDouble ? (kDblSlotCols > kSlotE + 4 * kEAtoms ? kDblSlotCols : kSlotE + 4 * kEAtoms)
                                               : kSlotE + 4 * kEAtoms;
  static constexpr int kSlots = (kTmemCols - kColSlots) / kSlotCols;    // caps the pipeline depth
  static_assert(kStageBytes % 1024 == 0 && kOffB % 1024 == 0, "operand tiles must keep 1024-byte alignment");
  static_assert(kAccStages * TILE_N <= kColSlots && kSlots >= 2, "tensor-memory column map overflows");
  static_assert(!kTailDouble || (kDblBytes <= kStageBytes && kDblOffB % 1024 == 0 && 2 * kTailN <= TILE_N),
                "a double tail stage must fit the ordinary stage");
  // the barriers take the first half of the barrier block, the per-stage item kinds sit in the second
  static_assert(8 * (4 * kMaxStages + 2 * kAccStages) + 16 <= kBarrierBytes / 2 && 4 * kMaxStages <= kBarrierBytes / 2,
                "barrier block overflows");
};

// Developer build only (-DPNV_WIDE_PROFILE): per-CTA cycle counters of the roles' waits, 16 per CTA, in a buffer
// read back with pnv_debug_wide_profile.  Not compiled into the library otherwise.
#ifdef PNV_WIDE_PROFILE
__device__ long long g_wide_prof[296 * 16];
#define PNV_PROF_T() clock64()
#define PNV_PROF_ACC(var, t0) var += clock64() - (t0)
#define PNV_PROF_SET(slot, v) g_wide_prof[blockIdx.x * 16 + (slot)] = (v)
#else
#define PNV_PROF_T() 0ll
#define PNV_PROF_ACC(var, t0) ((void)(t0), (void)(var))
#define PNV_PROF_SET(slot, v) ((void)(v))
#endif

__device__ __forceinline__ void named_bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// 16 bytes that this SM will not read again.
__device__ __forceinline__ void st_global_na(void* dst, const uint4& v) {
  asm volatile("st.global.L1::no_allocate.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

__device__ __forceinline__ uint64_t pack_desc(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

// Work items of an expert with c token rows: one per (token tile, M unit) - except that, with double tail items, the
// narrow tail tile (at most 64 live rows) takes one item per TWO M units.  full = the items of the ordinary tiles.
template <int TILE_N>
__device__ __forceinline__ unsigned expert_items(int c, int n_mu, bool dbl_tails, unsigned& full) {
  const unsigned nt = (unsigned)ceil_div_i(c, TILE_N);
  const bool tail = dbl_tails && c > 0 && c - (int)(nt - 1u) * TILE_N <= 64;
  full = (unsigned)n_mu * (nt - (tail ? 1u : 0u));
  return full + (tail ? (unsigned)(n_mu + 1) >> 1 : 0u);
}

// Work items position `unit` of `n_units` will process: items unit, unit + n_units, ... of the list every role
// walks.  Warp-collective.
template <int TILE_N>
__device__ __forceinline__ int my_work_items(const int* cnt, int E, int n_mu, bool dbl_tails, int unit, int n_units, int lane) {
  long long sum = 0;
  for (int e = lane; e < E; e += 32) {
    unsigned full;
    sum += expert_items<TILE_N>(cnt[e], n_mu, dbl_tails, full);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return (long long)unit < sum ? (int)((sum - unit + n_units - 1) / n_units) : 0;
}

// The work items of one unit (a CTA, or a CTA pair), in the order every role walks them: items unit, unit + units,
// ... of the (expert, token tile, M unit) order, so that units working at the same time share token rows through L2.
// next() moves to the following item and says whether there was one.
template <int TILE_N>
struct UnitTiles {
  int e, mu, nt;                 // the current item: expert, (first) M unit, token tile
  bool dbl;                      // ... a narrow tail tile against M units mu and mu + 1
  // 32-bit walk (the host bounds the item count of a launch).  `local` is the next item's index inside expert e_next,
  // `full` / `items` that expert's ordinary and total items; the division by the M units is a multiplication with the
  // rounded-down reciprocal and one correction (a hardware division takes a lone warp hundreds of cycles, and the
  // epilogue's share of a tile is short enough to feel that).
  const int* cnt;
  int E, n_mu, e_next;
  bool dbl_tails;
  unsigned local, step, full, items, inv_mu;
  __device__ void init(const int* s_counts, int E_, int n_mu_, bool dbl_tails_, int unit, int n_units) {
    cnt = s_counts; E = E_; n_mu = n_mu_; e_next = 0; dbl_tails = dbl_tails_; dbl = false;
    local = (unsigned)unit; step = (unsigned)n_units;
    inv_mu = n_mu > 1 ? (unsigned)(0x100000000ull / (unsigned)n_mu) : 0xFFFFFFFFu;
    items = expert_items<TILE_N>(cnt[0], n_mu, dbl_tails, full);
  }
  __device__ bool next() {
    while (local >= items) {
      local -= items;
      if (++e_next >= E) { e_next = E - 1; local = 0xFFFFFFFFu; items = 0; return false; }
      items = expert_items<TILE_N>(cnt[e_next], n_mu, dbl_tails, full);
    }
    if (local < full) {
      unsigned q = __umulhi(local, inv_mu), r = local - q * (unsigned)n_mu;
      if (r >= (unsigned)n_mu) { ++q; r -= (unsigned)n_mu; }
      nt = (int)q;
      mu = (int)r;
      dbl = false;
    } else {                      // (only with dbl_tails: otherwise full == items)
      nt = (cnt[e_next] - 1) / TILE_N;
      mu = 2 * (int)(local - full);
      dbl = true;
    }
    e = e_next;
    local += step;
    return true;
  }
};

// Does the tile at token offset n0 of an expert with cnt rows run as a narrow tail tile?
template <int TILE_N>
__device__ __forceinline__ bool narrow_tail(const Params& p, int cnt, int n0) {
  return TILE_N >= 128 && p.b_tail != 0 && cnt - n0 <= 64;
}

// One chunk of an accumulator (32 lanes of this warp's quarter x 8 * OCTETS token columns), scaled and rounded to bf16,
// as 8 x 8 fragments: pk[4 o + f] holds features 8 f .. 8 f + 7 of tokens 8 o .. 8 o + 7, two tokens to a register.
template <int OCTETS>
struct ChunkRegs {
  uint32_t lo[4 * OCTETS], hi[4 * OCTETS];      // accumulator lanes 0-15 and 16-31 of the quarter
};
__device__ __forceinline__ void chunk_load(uint32_t taddr, ChunkRegs<4>& c) {
  ptx::tc_ld_16x32(taddr, c.lo);
  ptx::tc_ld_16x32(taddr + (16u << 16), c.hi);
}
__device__ __forceinline__ void chunk_load(uint32_t taddr, ChunkRegs<2>& c) {
  ptx::tc_ld_16x16(taddr, c.lo);
  ptx::tc_ld_16x16(taddr + (16u << 16), c.hi);
}
__device__ __forceinline__ uint32_t scale_pack(float alpha, uint32_t a, uint32_t b) {
  const __nv_bfloat162 pr = __floats2bfloat162_rn(__fmul_rn(alpha, __uint_as_float(a)), __fmul_rn(alpha, __uint_as_float(b)));
  return *reinterpret_cast<const uint32_t*>(&pr);
}
template <int OCTETS>
__device__ __forceinline__ void chunk_pack(float alpha, const ChunkRegs<OCTETS>& c, uint32_t (&pk)[4 * OCTETS]) {
#pragma unroll
  for (int o = 0; o < OCTETS; ++o) {
    pk[4 * o] = scale_pack(alpha, c.lo[4 * o], c.lo[4 * o + 1]);
    pk[4 * o + 1] = scale_pack(alpha, c.lo[4 * o + 2], c.lo[4 * o + 3]);
    pk[4 * o + 2] = scale_pack(alpha, c.hi[4 * o], c.hi[4 * o + 1]);
    pk[4 * o + 3] = scale_pack(alpha, c.hi[4 * o + 2], c.hi[4 * o + 3]);
  }
}

template <int TILE_N, int STAGE_K, bool kFused, bool kPair, bool kDblTails>
__global__ void __launch_bounds__((4 + 16) * 32, 1)
group_mm_wide_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const __grid_constant__ CUtensorMap map_b_tail, const __grid_constant__ CUtensorMap map_out, const Params p) {
  using C = WideCfg<TILE_N, STAGE_K, kPair, kDblTails>;
  using Tiles = UnitTiles<TILE_N>;
  constexpr int kCtas = C::kCtas;
  constexpr int kChunk = C::kChunk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  uint8_t* after_stages = stage_base + p.stages * C::kStageBytes;
  uint8_t* s_out = after_stages;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(after_stages + C::kOutBytes);
  uint64_t* empty_bar = full_bar + C::kMaxStages;
  uint64_t* sf_full = empty_bar + C::kMaxStages;
  uint64_t* peer_full = sf_full + C::kMaxStages;
  uint64_t* acc_full = peer_full + C::kMaxStages;
  uint64_t* acc_empty = acc_full + C::kAccStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + C::kAccStages);
  // per pipeline stage: does it belong to a double tail item?  Written by the metadata producer before its
  // arrival on the stage's full barrier, read by the copiers after their wait on it.
  volatile int* s_kind = reinterpret_cast<volatile int*>(after_stages + C::kOutBytes + C::kBarrierBytes / 2);
  int* s_counts = reinterpret_cast<int*>(after_stages + C::kOutBytes + C::kBarrierBytes);

  float* s_alphas = reinterpret_cast<float*>(s_counts + p.E);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // position of this CTA (or CTA pair) in the work list, and of this CTA inside its pair
  const uint32_t rank = kPair ? ptx::cluster_ctarank() : 0u;
  const int unit = kPair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int n_units = kPair ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int n_mu = kPair ? (p.n_mt + 1) / 2 : p.n_mt;      // work items per token tile: M tiles, or pairs of them
  const bool dbl_tails = C::kTailDouble && p.b_tail != 0;  // narrow tail tiles take two M units per work item

  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
    ptx::prefetch_tensormap(&map_b_tail);
    if (!kFused && p.out_tma) ptx::prefetch_tensormap(&map_out);
    for (int s = 0; s < p.stages; ++s) {
      ptx::mbar_init(full_bar + s, 2);
      ptx::mbar_init(empty_bar + s, 1);
      ptx::mbar_init(sf_full + s, 1);
      ptx::mbar_init(peer_full + s, 1);
    }
    for (int a = 0; a < C::kAccStages; ++a) {
      ptx::mbar_init(acc_full + a, 1);
      ptx::mbar_init(acc_empty + a, C::kEpilogueWarps * kCtas);
    }
    ptx::fence_mbar_init();
  }
  if (warp == 2) {
    ptx::tmem_alloc<kCtas>(tmem_slot, kTmemCols);
    ptx::tmem_relinquish<kCtas>();
  }
  // counts (and everything else the producer kernels wrote) may only be read after this point
  pdl_wait();
  pdl_launch_dependents();
  for (int i = threadIdx.x; i < p.E; i += C::kThreads) {
    s_counts[i] = max(0, min(p.counts[i], p.max_n));
    s_alphas[i] = p.alphas[i];
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (kPair) ptx::cluster_sync();     // the partner's barriers are initialised before anything arrives on them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 2) {
    // =============================== producers ===============================
    const bool tile_role = warp == 0;
    Tiles tiles;
    tiles.init(s_counts, p.E, n_mu, dbl_tails, unit, n_units);
    bool ok = true;
    int stage = 0;
    uint32_t turn = 0;
    long long pf_wait = 0;
    while (ok && tiles.next()) {
      const int e = tiles.e;
      const int n0 = tiles.nt * TILE_N;
      // the second CTA of a pair takes the odd M tile; past the last tile it re-reads the last one (its
      // results are never stored), so every copy stays inside the expert's operands
      const int mt = kPair ? min(2 * tiles.mu + (int)rank, p.n_mt - 1) : tiles.mu;
      const bool tail = narrow_tail<TILE_N>(p, s_counts[e], n0);
      // a double tail item: the second M unit's tile (again clamped: past the last unit its results are dropped)
      const bool dbl = C::kTailDouble && tiles.dbl;
      const int mt1 = dbl ? min(2 * (tiles.mu + 1) + (int)rank, p.n_mt - 1) : mt;
      const uint8_t* sfb_base = p.sfb + (((long long)e * p.sfb_rt + (n0 >> 7)) * p.n_kt) * 512;
      const int sfb_row_atoms = (TILE_N > 128 && !tail) ? min(2, p.sfb_rt - (n0 >> 7)) : 1;
      const uint8_t* e_base = p.e_meta + (((long long)e * p.e_k_atoms) * p.e_m_atoms + mt) * 2048;
      const uint8_t* sfa_base = p.sfa + (((long long)e * p.n_mt + mt) * p.n_kt) * 512;
      const int nb = n0 + (int)rank * (tail ? C::kTailBRows : C::kBRows);      // this CTA's share of the token rows
#pragma unroll 1
      for (int ks = 0; ks < p.k_stages; ++ks) {
        const int k_atoms = min(C::kAtoms, p.n_kt - ks * C::kAtoms);
        const int b_boxes = (k_atoms + 1) / 2;
        const int e_atoms = (k_atoms + 1) / 2;
        const uint32_t sf_bytes = 512u * k_atoms;
        uint8_t* st = stage_base + stage * C::kStageBytes;
        const long long tp0 = PNV_PROF_T();
        if (!ptx::mbar_wait_warp(empty_bar + stage, turn ^ 1u)) {
          atomicExch(&g_status, tile_role ? kProducerEmptyTimeout : kSideProducerTimeout);
          ok = false;
          break;
        }
        PNV_PROF_ACC(pf_wait, tp0);                             // waiting for a free stage
        if (ptx::elect_one()) {
          if (tile_role) {
            // with the 4-D activation map one copy fetches all of the stage's 256-K chunks (a box past the
            // last chunk is zero-filled and still counts its full size)
            const uint32_t tile_bytes = (dbl ? 2 * C::kABytes : C::kABytes) +
                                        (p.b_4d ? C::kBBoxes : b_boxes) * (tail ? C::kTailBBoxBytes : C::kBBoxBytes);
            if (kPair) {
              // The tiles of BOTH CTAs are counted on the first CTA's barrier (the second CTA's loads name it as
              // theirs: .cta_group::2), so nothing has to relay "the big copies have landed" across the pair; the
              // first CTA expects both CTAs' bytes (the boxes are the same size), the second only arrives.
              if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar + stage, 2 * tile_bytes);
              else ptx::mbar_arrive(full_bar + stage);
              ptx::tma_load_3d_pair(st + C::kOffA, &map_a, full_bar + stage, 0, ks * C::kARowBytes, mt * kTileM, e);
              if (dbl) {              // both units' weights, then the one narrow activation box
                ptx::tma_load_3d_pair(st + C::kDblOffA1, &map_a, full_bar + stage, 0, ks * C::kARowBytes, mt1 * kTileM, e);
                ptx::tma_load_4d_pair(st + C::kDblOffB, &map_b_tail, full_bar + stage, 0, 0, nb, ks * C::kBBoxes, e);
              } else if (tail) {      // (only with the 4-D maps)
                ptx::tma_load_4d_pair(st + C::kOffB, &map_b_tail, full_bar + stage, 0, 0, nb, ks * C::kBBoxes, e);
              } else if (p.b_4d) {
                ptx::tma_load_4d_pair(st + C::kOffB, &map_b, full_bar + stage, 0, 0, nb, ks * C::kBBoxes, e);
              } else {
                for (int b = 0; b < b_boxes; ++b)
                  ptx::tma_load_3d_pair(st + C::kOffB + b * C::kBBoxBytes, &map_b, full_bar + stage, 0,
                                        ks * (STAGE_K / 2) + b * 128, nb, e);
              }
            } else {
              ptx::mbar_arrive_expect_tx(full_bar + stage, tile_bytes);
              ptx::tma_load_3d(st + C::kOffA, &map_a, full_bar + stage, ks * C::kARowBytes, mt * kTileM, e);
              if (tail) {             // (only with the 4-D maps)
                ptx::tma_load_4d(st + C::kOffB, &map_b_tail, full_bar + stage, 0, nb, ks * C::kBBoxes, e);
              } else if (p.b_4d) {
                ptx::tma_load_4d(st + C::kOffB, &map_b, full_bar + stage, 0, nb, ks * C::kBBoxes, e);
              } else {
                for (int b = 0; b < b_boxes; ++b)
                  ptx::tma_load_3d(st + C::kOffB + b * C::kBBoxBytes, &map_b, full_bar + stage,
                                   ks * (STAGE_K / 2) + b * 128, nb, e);
              }
            }
          } else {
            if (C::kTailDouble) s_kind[stage] = dbl ? 1 : 0;
            ptx::mbar_arrive_expect_tx(full_bar + stage, (dbl ? 2 : 1) * e_atoms * 2048 +
                                                             sf_bytes * (dbl ? 3 : 1 + sfb_row_atoms));
            for (int ea = 0; ea < e_atoms; ++ea) {
              const uint8_t* src = e_base + (long long)(ks * C::kEAtoms + ea) * p.e_m_atoms * 2048;
              if (dbl) {
                ptx::bulk_load(st + C::kDblOffE + ea * 2048, src, 2048, full_bar + stage);
                ptx::bulk_load(st + C::kDblOffE + C::kEBytes + ea * 2048, src + (mt1 - mt) * 2048, 2048, full_bar + stage);
              } else {
                ptx::bulk_load(st + C::kOffE + ea * 2048, src, 2048, full_bar + stage);
              }
            }
            const uint8_t* src = sfa_base + ks * (C::kAtoms * 512);
            if (dbl) {
              ptx::bulk_load(st + C::kDblOffSfa, src, sf_bytes, full_bar + stage);
              ptx::bulk_load(st + C::kDblOffSfa + C::kSfaBytes, src + (long long)(mt1 - mt) * p.n_kt * 512, sf_bytes, full_bar + stage);
              ptx::bulk_load(st + C::kDblOffSfb, sfb_base + (long long)(ks * C::kAtoms) * 512, sf_bytes, full_bar + stage);
            } else {
              ptx::bulk_load(st + C::kOffSfa, src, sf_bytes, full_bar + stage);
              for (int ra = 0; ra < sfb_row_atoms; ++ra)
                ptx::bulk_load(st + C::kOffSfb + ra * C::kSfaBytes,
                               sfb_base + ((long long)ra * p.n_kt + ks * C::kAtoms) * 512, sf_bytes, full_bar + stage);
            }
          }
        }
        __syncwarp();
        if (++stage == p.stages) { stage = 0; turn ^= 1u; }
      }
    }
    if (threadIdx.x == 0) PNV_PROF_SET(0, pf_wait);
    if (!ok) {
      // give copies already in flight time to land before the CTA's shared memory is released
#pragma unroll 1
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 2) {
    // =============================== MMA issuer ===============================
    const int n_items = my_work_items<TILE_N>(s_counts, p.E, n_mu, dbl_tails, unit, n_units, lane);
    if (rank == 0) {
      constexpr uint32_t idesc_full = ptx::mma_sp_nvf4_idesc(TILE_N, kTileM * kCtas);
      constexpr uint32_t idesc_tail = ptx::mma_sp_nvf4_idesc(C::kTailN, kTileM * kCtas);
      Tiles tiles;
      tiles.init(s_counts, p.E, n_mu, dbl_tails, unit, n_units);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0, soff = 0;
      bool ok = true;
      // first-tile descriptors, split into the 32-bit halves: only the low half changes with the address
      const uint64_t d_a0 = ptx::smem_desc(ptx::smem_u32(stage_base) + C::kOffA, 8 * C::kARowBytes, 16, C::kASwizzle);
      const uint64_t d_b0 = ptx::smem_desc(ptx::smem_u32(stage_base) + C::kOffB, 1024, 16, 2);
      const uint32_t lo_a0 = (uint32_t)d_a0, hi_a = (uint32_t)(d_a0 >> 32);
      const uint32_t lo_b0 = (uint32_t)d_b0, hi_b = (uint32_t)(d_b0 >> 32);
      const uint32_t slots0 = tmem_base + C::kColSlots;
      const int last_atoms = p.n_kt - (p.k_stages - 1) * C::kAtoms;     // K-blocks of a tile's last stage
      const long long ti0 = PNV_PROF_T();
      long long pf_acc = 0, pf_slot = 0, pf_issue = 0, pf_loop = 0;
      for (int item = 0; item < n_items && ok; ++item) {
        // a 64-wide tile's scales sit 0 or 2 columns into the 128-row atom (even offsets only: the MMA
        // faults on an odd scale column); wider tiles start at column 0 and need no tile coordinates
        uint32_t sfb_off = 0;
        uint32_t idesc = idesc_full, bbox16 = C::kBBoxBytes >> 4;
        bool dbl = false;
        if (TILE_N < 128 || p.b_tail != 0) {
          if (!tiles.next()) break;
          if (TILE_N < 128) sfb_off = ((tiles.nt * TILE_N) & 127) >> 5;
          if (narrow_tail<TILE_N>(p, s_counts[tiles.e], tiles.nt * TILE_N)) {
            idesc = idesc_tail;
            bbox16 = C::kTailBBoxBytes >> 4;
            dbl = C::kTailDouble && tiles.dbl;
          }
        }
        const long long ta0 = PNV_PROF_T();
        if (!ptx::mbar_wait_warp(acc_empty + acc, acc_phase ^ 1)) {
          atomicExch(&g_status, kMmaAccTimeout);
          ok = false;
          break;
        }
        PNV_PROF_ACC(pf_acc, ta0);                              // waiting for a free accumulator
        ptx::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TILE_N;
        // The K loop of one item, compiled twice (ordinary items; double tail items) and chosen per item: whatever
        // the issuing thread executes between two MMAs is time the tensor pipe waits for, so the loop of an ordinary
        // item carries nothing of the other kind.
        auto item_stages = [&](auto dbl_kind, auto full_kind) {
          constexpr bool kDbl = decltype(dbl_kind)::value;
          constexpr bool kFull = decltype(full_kind)::value;      // K is a whole number of stages: no short last stage
#pragma unroll 1
          for (int ks = 0; ks < p.k_stages; ++ks) {
            const int k_atoms = kFull ? C::kAtoms : ks + 1 == p.k_stages ? last_atoms : C::kAtoms;
            const long long ts0 = PNV_PROF_T();
            if (!ptx::mbar_wait_warp(sf_full + stage, phase)) {
              atomicExch(&g_status, kMmaScaleTimeout);
              ok = false;
              break;
            }
            PNV_PROF_ACC(pf_slot, ts0);                           // waiting for a filled slot (own tiles)
            ptx::tc_fence_after();
            const long long tm0 = PNV_PROF_T();
            // descriptors of this stage: the precomputed ones of stage 0 plus the stage's offset in
            // 16-byte units (the address field is the low 14 bits, so a 32-bit add cannot carry out)
            const uint32_t la = lo_a0 + soff, lb = lo_b0 + soff;
            const uint32_t slot = slots0 + stage * C::kSlotCols;
            if (ptx::elect_one()) {
            if constexpr (kDbl) {
              // a narrow tail tile against two M units: the units' weights sit kABytes apart, their accumulators
              // kTailN columns apart, and both read the one activation box and its scales
              const uint32_t lbd = lb + ((C::kDblOffB - C::kOffB) >> 4);
#pragma unroll
              for (int ka = 0; ka < C::kAtoms; ++ka) {
                if (ka < k_atoms) {
                  const uint64_t db = pack_desc(lbd + (ka >> 1) * (C::kTailBBoxBytes >> 4) + (ka & 1) * 4, hi_b);
                  const uint32_t sfb_d = slot + C::kDblSlotSfb + ka * 4;
                  ptx::tc_mma_sp_nvf4<kCtas>(d_tmem, pack_desc(la + ka * 2, hi_a), db, idesc_tail, (ks | ka) != 0 ? 1u : 0u,
                                             slot + ka * 4, sfb_d, slot + C::kDblSlotE + ka * 2);
                  ptx::tc_mma_sp_nvf4<kCtas>(d_tmem + C::kTailN, pack_desc(la + (C::kDblOffA1 >> 4) + ka * 2, hi_a), db,
                                             idesc_tail, (ks | ka) != 0 ? 1u : 0u, slot + C::kDblSlotSfa1 + ka * 4, sfb_d,
                                             slot + C::kDblSlotE1 + ka * 2);
                }
              }
            } else {
              const uint32_t sfb_cols = slot + C::kSlotSfb + sfb_off;
#pragma unroll
              for (int ka = 0; ka < C::kAtoms; ++ka)
                if (kFull || ka < k_atoms)
                  ptx::tc_mma_sp_nvf4<kCtas>(d_tmem, pack_desc(la + ka * 2, hi_a),
                                             pack_desc(lb + (ka >> 1) * bbox16 + (ka & 1) * 4, hi_b), idesc,
                                             ka != 0 ? 1u : ks != 0 ? 1u : 0u, slot + ka * 4,
                                             sfb_cols + ka * C::kSfbColsPerAtom, slot + C::kSlotE + ka * 2);
            }
            // shared-memory stage and tensor-memory slot reusable (in both CTAs of a pair) once these MMAs retire
            ptx::tc_commit_n<kCtas>(empty_bar + stage);
            if (ks + 1 == p.k_stages) ptx::tc_commit_n<kCtas>(acc_full + acc);
            }
            __syncwarp();
            PNV_PROF_ACC(pf_issue, tm0);                          // issuing MMAs + commit
            soff += C::kStageBytes >> 4;
            if (++stage == p.stages) { stage = 0; soff = 0; phase ^= 1; }
          }
        };
        if (C::kTailDouble && dbl) item_stages(std::true_type{}, std::false_type{});
        else if (last_atoms == C::kAtoms) item_stages(std::false_type{}, std::true_type{});
        else item_stages(std::false_type{}, std::false_type{});
        if (!ok) break;
        if (++acc == C::kAccStages) { acc = 0; acc_phase ^= 1; }
      }
      PNV_PROF_ACC(pf_loop, ti0);
      PNV_PROF_SET(1, pf_acc); PNV_PROF_SET(2, pf_slot); PNV_PROF_SET(3, pf_issue); PNV_PROF_SET(4, pf_loop);
      PNV_PROF_SET(5, (long long)n_items * p.k_stages);
    }
    __syncwarp();
  } else if (warp == 3) {
    // =============================== copier ===============================
    // Every pipeline stage's scale and metadata atoms go from shared memory into the stage's slot of the ring in tensor
    // memory; the commit on the stage's sf_full barrier arrives once they are there.  Without double tail items the
    // copier does not walk the tiles: a narrow tail tile loads one activation-scale row atom instead of two, and the
    // copy of the other (whatever an older stage left there) lands in columns its 64-token MMAs never read.
    const int n_items = my_work_items<TILE_N>(s_counts, p.E, n_mu, dbl_tails, unit, n_units, lane);
    const long long n_stages = (long long)n_items * p.k_stages;
    // the second CTA of a pair only tells the first one when each stage's side copies have landed
    const bool relay = rank != 0;
    const uint64_t d_st0 = ptx::smem_desc(ptx::smem_u32(stage_base), 128, 0, 0);
    const uint32_t lo_st0 = (uint32_t)d_st0, hi = (uint32_t)(d_st0 >> 32);      // the descriptors differ in the address only
    const uint32_t slots0 = tmem_base + C::kColSlots;
    const int last_atoms = p.n_kt - (p.k_stages - 1) * C::kAtoms;
    const bool whole_stages = last_atoms == C::kAtoms;
    int stage = 0, ks = 0;
    uint32_t phase = 0;
    long long pf_cwait = 0, pf_cissue = 0;
    bool dbl = false;       // a double tail item's stages are laid out differently: the producer says which they are
#pragma unroll 1
    for (long long g = 0; g < n_stages; ++g) {
      const long long tc0 = PNV_PROF_T();
      if (!ptx::mbar_wait_warp(full_bar + stage, phase) || (kPair && !relay && !ptx::mbar_wait_warp(peer_full + stage, phase))) {
        atomicExch(&g_status, kScaleLoaderTimeout);
        break;
      }
      PNV_PROF_ACC(pf_cwait, tc0);                            // waiting for landed copies
      if (relay) {
        if (ptx::elect_one()) ptx::mbar_arrive_cluster(peer_full + stage, 0);
        __syncwarp();
      } else {
        if (C::kTailDouble && dbl_tails && ks == 0) dbl = s_kind[stage] != 0;
        ptx::tc_fence_after();
        const long long tc1 = PNV_PROF_T();
        const uint32_t lo = lo_st0 + (uint32_t)stage * (C::kStageBytes >> 4);
        const uint32_t slot = slots0 + stage * C::kSlotCols;
        // (compiled twice: K a whole number of stages, so that no copy needs a guard; or a short last stage)
        auto copy_stage = [&](auto full_kind) {
          constexpr bool kFull = decltype(full_kind)::value;
          const int k_atoms = kFull ? C::kAtoms : ks + 1 == p.k_stages ? last_atoms : C::kAtoms;
          if (C::kTailDouble && dbl) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
              for (int ka = 0; ka < C::kAtoms; ++ka)
                if (kFull || ka < k_atoms)
                  ptx::tc_cp_32x128b_warpx4<kCtas>(slot + u * C::kDblSlotSfa1 + ka * 4,
                                                   pack_desc(lo + ((C::kDblOffSfa + u * C::kSfaBytes) >> 4) + ka * 32, hi));
#pragma unroll
              for (int ea = 0; ea < C::kEAtoms; ++ea)
                if (kFull || 2 * ea < k_atoms)
                  ptx::tc_cp_128x128b<kCtas>(slot + C::kDblSlotE + u * (C::kDblSlotE1 - C::kDblSlotE) + ea * 4,
                                             pack_desc(lo + ((C::kDblOffE + u * C::kEBytes) >> 4) + ea * 128, hi));
            }
#pragma unroll
            for (int ka = 0; ka < C::kAtoms; ++ka)
              if (kFull || ka < k_atoms)
                ptx::tc_cp_32x128b_warpx4<kCtas>(slot + C::kDblSlotSfb + ka * 4, pack_desc(lo + (C::kDblOffSfb >> 4) + ka * 32, hi));
          } else {
#pragma unroll
            for (int ka = 0; ka < C::kAtoms; ++ka) {
              if (kFull || ka < k_atoms) {
                ptx::tc_cp_32x128b_warpx4<kCtas>(slot + ka * 4, pack_desc(lo + (C::kOffSfa >> 4) + ka * 32, hi));
#pragma unroll
                for (int ra = 0; ra < C::kSfbRowAtoms; ++ra)
                  ptx::tc_cp_32x128b_warpx4<kCtas>(slot + C::kSlotSfb + ka * C::kSfbColsPerAtom + ra * 4,
                                                   pack_desc(lo + ((C::kOffSfb + ra * C::kSfaBytes) >> 4) + ka * 32, hi));
              }
            }
#pragma unroll
            for (int ea = 0; ea < C::kEAtoms; ++ea)
              if (kFull || 2 * ea < k_atoms)
                ptx::tc_cp_128x128b<kCtas>(slot + C::kSlotE + ea * 4, pack_desc(lo + (C::kOffE >> 4) + ea * 128, hi));
          }
        };
        if (ptx::elect_one()) {
          if (whole_stages) copy_stage(std::true_type{});
          else copy_stage(std::false_type{});
          ptx::tc_commit_local<kCtas>(sf_full + stage);     // arrives once the copies above have completed
        }
        __syncwarp();
        PNV_PROF_ACC(pf_cissue, tc1);                           // issuing copies
      }
      if (++ks == p.k_stages) ks = 0;
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    if (!relay) { PNV_PROF_SET(6, pf_cwait); PNV_PROF_SET(7, pf_cissue); }
    __syncwarp();
  } else {
    // =============================== epilogue ===============================
    const int group = (warp - C::kFirstEpilogueWarp) >> 2;   // chunks of kChunk token columns are dealt to the four groups in turn
    const int sub = warp & 3;                  // tensor-memory lane quarter this warp may read
    const int gwarp = (warp - C::kFirstEpilogueWarp) & 3;    // this warp's place in its group
    uint8_t* gbuf = s_out + group * 8192;      // the group's staging area
    const bool wide_rows = (p.M & 7) == 0;     // output rows are 16-byte aligned
    int acc = 0;
    uint32_t acc_phase = 0;
    if (kFused) {
      // Benign fill of GEMM2's scale buffer: every byte the epilogues will not write (rows at or
      // past counts[e], K-block slop) becomes 0x38.  All CTAs share the lines; live slots are
      // skipped, so the fill never races with a quantized scale.
      const int KB = p.f_n / kSfBlock;
      const unsigned lines = (unsigned)p.E * p.sfb_rt * p.f_n_kt * 32u;   // < 2^27, checked by the host
      const uint32_t w4 = kBenignSf * 0x01010101u;
      constexpr unsigned kFillThreads = C::kEpilogueWarps * 32;
#pragma unroll 1
      for (unsigned c = blockIdx.x * kFillThreads + (threadIdx.x - C::kFirstEpilogueWarp * 32); c < lines; c += gridDim.x * kFillThreads) {
        const int rr = (int)(c & 31);
        unsigned a = c >> 5;
        const unsigned a_kt = a / (unsigned)p.f_n_kt;
        const int kt = (int)(a - a_kt * p.f_n_kt);
        const unsigned a_e = a_kt / (unsigned)p.sfb_rt;
        const int r0 = (int)(a_kt - a_e * p.sfb_rt) * 128 + rr;
        const int cnt_e = s_counts[a_e];
        uint8_t* line = p.f_sfb_out + (long long)c * 16;
        if (r0 >= cnt_e) {
          *reinterpret_cast<uint4*>(line) = make_uint4(w4, w4, w4, w4);
        } else {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (r0 + 32 * g >= cnt_e) {
              *reinterpret_cast<uint32_t*>(line + 4 * g) = w4;
            } else {
              for (int j = KB - kt * 4; j < 4; ++j)
                if (j >= 0) line[4 * g + j] = (uint8_t)kBenignSf;
            }
          }
        }
      }
    }
    // A warp hands its accumulator stage back as soon as it has read its last chunk of it (of a pair: to the
    // first CTA, where the issuers wait).
    auto release_acc = [&]() {
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (kPair && rank != 0) ptx::mbar_arrive_cluster(acc_empty + acc, 0);
        else ptx::mbar_arrive(acc_empty + acc);
      }
    };
    long long pf_ewait = 0, pf_ework = 0;
    Tiles tiles;
    tiles.init(s_counts, p.E, n_mu, dbl_tails, unit, n_units);
    while (tiles.next()) {
      // A double tail item holds two M units' 64-column accumulators side by side: epilogue groups 0-1 take the
      // first unit's two chunks, groups 2-3 the second unit's.
      const bool dbl = C::kTailDouble && tiles.dbl;
      const int e = tiles.e, mu = tiles.mu + (dbl ? group >> 1 : 0), nt = tiles.nt;
      const int chunk0 = dbl ? group & 1 : group;          // this group's first chunk of token columns
      const int cnt = s_counts[e];
      const int mt = kPair ? 2 * mu + (int)rank : mu;
      // the second CTA of the last pair of an odd tile count stores nothing, nor does anyone for a double item's
      // second unit past the last one
      const bool mt_valid = mt < p.n_mt;
      const float alpha = s_alphas[e];
      const float gs = kFused ? (p.f_gpe ? p.f_gscale[e] : p.f_gscale[0]) : 0.f;      // in flight while the warp waits
      const int n0 = nt * TILE_N;
      const long long te0 = PNV_PROF_T();
      if (!ptx::mbar_wait(acc_full + acc, acc_phase)) {
        atomicExch(&g_status, kEpilogueTimeout);
        break;
      }
      PNV_PROF_ACC(pf_ewait, te0);                              // waiting for an accumulator
      const long long te1 = PNV_PROF_T();
      ptx::tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(sub * 32) << 16) + acc * TILE_N + (dbl ? (group >> 1) * C::kTailN : 0);
      // Both of a warp's chunks leave tensor memory, scaled and packed to bf16, and the accumulator goes back to the
      // issuers before anything else is done with them: with one accumulator stage the tensor pipe waits that long.
      constexpr int kOwn = TILE_N / (4 * kChunk);         // chunks of a tile each group takes (1, or 2 for 256 tokens)
      constexpr int kOct = kChunk / 8;
      uint32_t pk[kOwn][4 * kOct];
      {
        ChunkRegs<kOct> v[kOwn];
        bool live[kOwn];
#pragma unroll
        for (int j = 0; j < kOwn; ++j) {
          const int c0 = (chunk0 + 4 * j) * kChunk;
          live[j] = mt_valid && n0 + c0 < cnt;
          if (live[j]) {
            chunk_load(t_row + c0, v[j]);
            ptx::tc_ld_wait();
            chunk_pack<kOct>(alpha, v[j], pk[j]);
          }
        }
      }
      release_acc();
#pragma unroll
      for (int j = 0; j < kOwn; ++j) {
        const int c0 = (chunk0 + 4 * j) * kChunk;
        const int rows = cnt - (n0 + c0);                 // live token rows from c0 on; the same for all lanes
        if (!mt_valid || rows <= 0) break;                // uniform over the group
        if (!kFused) {
          // Plain epilogue.  The group's four warps lay their 32 features side by side in shared memory ([64-feature
          // half][token][128 bytes], 16-byte pieces swizzled by the token so that nobody has bank conflicts; the
          // transpose is stmatrix's).  A chunk whose token rows are all live leaves as two TMA stores; in any other
          // case every store instruction writes 256 contiguous bytes of two output rows, and rows at or past counts[e]
          // are skipped.
          const bool whole = p.out_tma != 0 && rows >= kChunk;
          if (p.out_tma != 0 && gwarp == 0) {             // the previous chunk's TMA stores have read the area
            if (ptx::elect_one()) ptx::bulk_wait_read_all();
            __syncwarp();
          }
          named_bar_sync(1 + group, 128);                 // ... and so has the group
          {
            const int t = lane & 7, c = (sub & 1) * 4 + (lane >> 3);
            const uint32_t dst = ptx::smem_u32(gbuf) + (sub >> 1) * (kChunk * 128) + t * 128 + ((c ^ t) << 4);
#pragma unroll
            for (int o = 0; o < kOct; ++o)
              ptx::stmatrix_x4_trans(dst + o * 1024, pk[j][4 * o], pk[j][4 * o + 1], pk[j][4 * o + 2], pk[j][4 * o + 3]);
          }
          if (whole) ptx::fence_proxy_async_smem();
          named_bar_sync(1 + group, 128);
          if (whole) {
            if (gwarp == 0) {
              if (ptx::elect_one()) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                  if (mt * kTileM + h * 64 < p.M)
                    ptx::tma_store_3d(&map_out, gbuf + h * (kChunk * 128), mt * kTileM + h * 64, n0 + c0, e);
                ptx::bulk_commit();
              }
              __syncwarp();
            }
            continue;
          }
          const int piece = lane & 15;
          const int m8 = mt * kTileM + piece * 8;
          const long long src_row = (long long)e * p.max_n + n0 + c0;
#pragma unroll
          for (int i = 0; i < kOct; ++i) {
            const int t = gwarp * 2 + (lane >> 4) + 8 * i;
            if (t < rows && m8 < p.M) {
              __nv_bfloat16* d = nullptr;
              if (p.row_map == nullptr) {
                d = p.out + (src_row + t) * p.M + m8;
              } else {
                const int to = p.row_map[src_row + t];
                if (to >= 0) d = mapped_row(p, to) + m8;
              }
              if (d != nullptr) {
                const uint4 x = *reinterpret_cast<const uint4*>(gbuf + (piece >> 3) * (kChunk * 128) + t * 128 + (((piece & 7) ^ (t & 7)) << 4));
                if (wide_rows) {
                  st_global_na(d, x);
                } else {                                  // rows that are not 16-byte aligned, element by element
                  unsigned short* h = reinterpret_cast<unsigned short*>(d);
                  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                  for (int q = 0; q < 8; ++q)
                    if (m8 + q < p.M) h[q] = (unsigned short)(w[q >> 1] >> (16 * (q & 1)));
                }
              }
            }
          }
        } else {
          // Fused epilogue.  The weight rows are interleaved in 64-row blocks (32 gate rows, then the 32 matching up
          // rows), so of a warp pair (lane quarters 0-1 or 2-3) one warp holds the gates and the other the ups of the
          // same 32 output features: exactly one quantization block per token.  Both transpose their values into the
          // pair's buffer ([token][gates 64 bytes | ups 64 bytes], pieces swizzled as above); then a thread takes half
          // a block of one token - 16 features, so 64 threads share the chunk - and everything is in its registers:
          // activation, amax (one exchange with the lane that has the other half), scale, codes.
          const bool is_up = (sub & 1) != 0;
          const int par = is_up ? 1 : 0;
          uint8_t* pbuf = gbuf + (sub >> 1) * 4096;
          const int pair_bar = 1 + group * 2 + (sub >> 1);
          constexpr int kTw = kChunk / 2;                   // tokens a warp of the pair finishes
          named_bar_sync(pair_bar, 64);                     // the pair has read the previous chunk
          {
            const int t = lane & 7, c = par * 4 + (lane >> 3);
            const uint32_t dst = ptx::smem_u32(pbuf) + t * 128 + ((c ^ t) << 4);
#pragma unroll
            for (int o = 0; o < kOct; ++o)
              ptx::stmatrix_x4_trans(dst + o * 1024, pk[j][4 * o], pk[j][4 * o + 1], pk[j][4 * o + 2], pk[j][4 * o + 3]);
          }
          named_bar_sync(pair_bar, 64);
          const int t = par * kTw + (lane & (kTw - 1));     // this lane's token inside the chunk
          const int half = (lane / kTw) & 1;                // which 16 features of the block
          const bool work = lane < 2 * kTw && t < rows;
          uint32_t y[8];                                    // results, two features to a register
          {
            const uint8_t* row = pbuf + t * 128;
            const uint4 g0 = *reinterpret_cast<const uint4*>(row + (((2 * half) ^ (t & 7)) << 4));
            const uint4 g1 = *reinterpret_cast<const uint4*>(row + (((2 * half + 1) ^ (t & 7)) << 4));
            const uint4 u0 = *reinterpret_cast<const uint4*>(row + (((2 * half + 4) ^ (t & 7)) << 4));
            const uint4 u1 = *reinterpret_cast<const uint4*>(row + (((2 * half + 5) ^ (t & 7)) << 4));
            const uint32_t g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
            const uint32_t u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
            gated_act16(g, u, p.f_act, y);
          }
          uint32_t m = bf16x2_amax8(y);
          m = bf16x2_max(m, __shfl_xor_sync(0xffffffffu, m, kTw));
          const float amax = fmaxf(fmaxf(bf16_lo(m), bf16_hi(m)), 0.f);
          if (work) {
            uint32_t sf_byte;
            float inv;
            block_scale(amax, gs, sf_byte, inv);
            const int kb = mt * 2 + (sub >> 1);             // 32-feature block of the N-wide output
            const int n = n0 + c0 + t;
            const long long row = (long long)e * p.max_n + n;
            *reinterpret_cast<uint2*>(p.f_b_out + row * (p.f_n / 2) + kb * 16 + half * 8) =
                make_uint2(quant8_packed(y[0], y[1], y[2], y[3], inv), quant8_packed(y[4], y[5], y[6], y[7], inv));
            if (half == 0) p.f_sfb_out[sf_offset(e, n, kb, p.sfb_rt, p.f_n_kt)] = (uint8_t)sf_byte;
          }
        }
      }
      PNV_PROF_ACC(pf_ework, te1);                              // this group's share of the tile
      if (++acc == C::kAccStages) { acc = 0; acc_phase ^= 1; }
    }
    if (!kFused && p.out_tma != 0 && gwarp == 0) {         // the last stores are done with shared memory
      if (ptx::elect_one()) ptx::bulk_wait_all();
      __syncwarp();
    }
    if (group == 0 && sub == 0 && lane == 0) { PNV_PROF_SET(8, pf_ewait); PNV_PROF_SET(9, pf_ework); }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (kPair) ptx::cluster_sync();     // the partner has stopped reading this CTA's shared and tensor memory
  if (warp == 2) {
    __syncwarp();
    ptx::tc_fence_after();
    ptx::tmem_dealloc<kCtas>(tmem_base, kTmemCols);
  }
}
