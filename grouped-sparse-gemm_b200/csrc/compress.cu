// Load-time weight compressor: dense packed e2m1 [E, M, K/2] + natural-order UE4M3 [E, M, K/32]
// -> the three operands the sparse block-scaled MMA reads:
//   a_comp  [E, M, round_up(K,64)/4]   the two kept bytes (e2m1 pairs) of every 4-byte chunk
//   e_meta  [E, round_up(M,128), round_up(K,256)/16]  one nibble per chunk = the two 2-bit
//           in-chunk indices of the kept bytes, in 128-row x 16-byte atoms (see common.cuh)
//   sfa     swizzled scale atoms, slop bytes zero
//
// Bound: HBM (one layer's 8 x 28672 x 4096 weights: 499 MB in, 323 MB out, 126 us at the measured copy rate of 6.55 TB/s).  One kernel, a block per
// tile of 128 rows x 1024 K: a lane reads 32 bytes (8 chunks), emits 16 bytes of a_comp and 4 bytes of metadata, a quad of
// lanes owns one (row, 256-K) metadata line, and a lane has four lines in flight; then a lane per 16-byte line of the
// tile's scale atoms.  The divisions that place a tile are made once per block, and a chunk costs about 15 instructions
// without branches.  With per-lane 64-bit divisions, a data-dependent select loop per chunk and byte-sized scale loads in a
// second kernel these weights took 1166 us, now 128 to 133.
#include "common.cuh"

namespace pnv {
namespace {

constexpr int kThreads = 256;
constexpr int kTileLines = 4;            // 256-K metadata lines of a tile along K

// Non-zero mask of a chunk's four bytes (bit i = byte i) -> the two 2-bit in-chunk indices of the kept bytes: the first two
// non-zero ones; a lone byte is paired with a zero so that the indices stay strictly ordered ((byte @i, 0 @3) for
// i < 3, (0 @0, byte @3) for i = 3); an empty chunk gives (0, 0).
__host__ __device__ constexpr uint32_t chunk_nibble(uint32_t mask) {
  uint32_t first = 4, second = 4;
  for (uint32_t i = 0; i < 4; ++i) {
    if ((mask >> i & 1u) == 0) continue;
    if (first == 4) first = i;
    else if (second == 4) second = i;
  }
  if (first == 4) return 0;
  if (second == 4) return first == 3 ? 0u | (3u << 2) : first | (3u << 2);
  return first | (second << 2);
}
__host__ __device__ constexpr uint64_t chunk_nibbles() {
  uint64_t t = 0;
  for (uint32_t m = 0; m < 16; ++m) t |= (uint64_t)chunk_nibble(m) << (4 * m);
  return t;
}

// Two 4-byte chunks (16 e2m1 values) -> their four kept bytes and two index nibbles.  A byte is "zero" when both its
// magnitudes are zero; such bytes are cleared (sign bits too) so that a padding index finds a zero byte.
__device__ __forceinline__ uint32_t compress_pair(uint32_t c0, uint32_t c1, uint32_t& nibbles) {
  constexpr uint64_t kTable = chunk_nibbles();
  // bit 0 of every byte: is it non-zero (magnitude bits are 0x77, so the sum cannot carry into the next byte)
  const uint32_t z0 = (((c0 & 0x77777777u) + 0x7F7F7F7Fu) >> 7) & 0x01010101u;
  const uint32_t z1 = (((c1 & 0x77777777u) + 0x7F7F7F7Fu) >> 7) & 0x01010101u;
  // the four bits side by side at the top (the other partial products fall on distinct lower bits), times 4
  const uint32_t n0 = (uint32_t)(kTable >> ((z0 * 0x10204080u) >> 26 & 0x3Cu)) & 15u;
  const uint32_t n1 = (uint32_t)(kTable >> ((z1 * 0x10204080u) >> 26 & 0x3Cu)) & 15u;
  nibbles = n0 | (n1 << 4);
  const uint32_t both = n0 | (n1 << 8);
  const uint32_t sel = ((both | (both << 2)) & 0x3333u) | 0x4400u;      // byte selectors: first chunk 0-3, second 4-7
  return __byte_perm(c0 & (z0 * 255u), c1 & (z1 * 255u), sel);
}

__global__ void __launch_bounds__(kThreads)
compress_kernel(const uint8_t* __restrict__ w_packed, const uint8_t* __restrict__ sf_nat, long long tiles, int M, int K,
                WeightDims wd, uint8_t* __restrict__ a_comp, uint8_t* __restrict__ e_meta, uint8_t* __restrict__ sfa) {
  const int k_atoms = wd.k_e / 16;            // 256-K metadata atoms per row
  const int m_atoms = wd.m_e / 128;
  const int row_bytes_in = K / 2;
  const int row_bytes_ac = wd.k_ac / 2;
  const int KB = ceil_div_i(K, kSfBlock), n_kt = sf_k_atoms(K);
  const unsigned k_tiles = (unsigned)ceil_div_i(k_atoms, kTileLines);
  const bool vec_in = (row_bytes_in % 16) == 0 && (reinterpret_cast<uintptr_t>(w_packed) % 16) == 0;
  const bool vec_sf = (KB % 4) == 0 && (reinterpret_cast<uintptr_t>(sf_nat) % 4) == 0;
  const int q = threadIdx.x & 3;              // which 64-K quarter of a 256-K line
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long row_tile = tile / k_tiles;                    // e * m_atoms + row atom
    const int ka0 = (int)(tile - row_tile * k_tiles) * kTileLines;
    const int e = (int)(row_tile / m_atoms);
    const int m_base = (int)(row_tile - (long long)e * m_atoms) * 128;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int mr = half * 64 + (threadIdx.x >> 2);              // row of the tile
      const int m = m_base + mr;
      const uint8_t* src = w_packed + ((long long)e * M + m) * row_bytes_in + ka0 * 128 + q * 32;
      uint32_t in[kTileLines][8];
#pragma unroll
      for (int i = 0; i < kTileLines; ++i) {
        const int kbyte0 = (ka0 + i) * 128 + q * 32;              // first input byte of this lane's piece
        if (m < M && vec_in && kbyte0 + 32 <= row_bytes_in) {
          const uint4 v0 = __ldg(reinterpret_cast<const uint4*>(src + i * 128));
          const uint4 v1 = __ldg(reinterpret_cast<const uint4*>(src + i * 128) + 1);
          in[i][0] = v0.x; in[i][1] = v0.y; in[i][2] = v0.z; in[i][3] = v0.w;
          in[i][4] = v1.x; in[i][5] = v1.y; in[i][6] = v1.z; in[i][7] = v1.w;
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c)         // K % 8 == 0, so whole 4-byte chunks exist or not
            in[i][c] = (m < M && kbyte0 + c * 4 + 4 <= row_bytes_in) ? __ldg(reinterpret_cast<const uint32_t*>(src + i * 128) + c) : 0u;
        }
      }
#pragma unroll
      for (int i = 0; i < kTileLines; ++i) {
        const int ka = ka0 + i;
        if (ka >= k_atoms) break;
        uint32_t out[4], meta = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t nib;
          out[c] = compress_pair(in[i][2 * c], in[i][2 * c + 1], nib);
          meta |= nib << (8 * c);
        }
        // metadata line: atom (e, ka, m / 128), row m % 128, 4 bytes per lane; zero for rows past M
        const long long atom = ((long long)e * k_atoms + ka) * m_atoms + (m_base >> 7);
        *reinterpret_cast<uint32_t*>(e_meta + atom * 2048 + mr * 16 + q * 4) = meta;
        const int acbyte0 = ka * 64 + q * 16;
        if (m < M && acbyte0 < row_bytes_ac)
          *reinterpret_cast<uint4*>(a_comp + ((long long)e * wd.m_ac + m) * row_bytes_ac + acbyte0) =
              make_uint4(out[0], out[1], out[2], out[3]);
      }
    }
    // the tile's scales: 8 K-atoms x 32 lines of 16 bytes (rows rr, rr + 32, rr + 64, rr + 96), slop bytes zero
    static_assert(kTileLines * 2 * 32 == kThreads, "one scale line per thread");
    const int kt = ka0 * 2 + (int)(threadIdx.x & 7), rr = (int)(threadIdx.x >> 3);
    if (kt < n_kt) {
      uint32_t w[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int m = m_base + rr + 32 * g;
        const uint8_t* src = sf_nat + ((long long)e * M + m) * KB + kt * 4;
        w[g] = 0u;
        if (m < M) {
          if (vec_sf) {
            w[g] = __ldg(reinterpret_cast<const uint32_t*>(src));
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (kt * 4 + i < KB) w[g] |= (uint32_t)__ldg(src + i) << (8 * i);
          }
        }
      }
      *reinterpret_cast<uint4*>(sfa + (row_tile * n_kt + kt) * 512 + rr * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

}  // namespace
}  // namespace pnv

using namespace pnv;

extern "C" int pnv_compress(const uint8_t* w_packed, const uint8_t* w_blockscale, int experts,
                            int features, int k, uint8_t* a_comp, uint8_t* e_meta, uint8_t* sfa,
                            pnv_stream_t stream) {
  PNV_REQUIRE(w_packed && w_blockscale && a_comp && e_meta && sfa, "null pointer argument");
  PNV_REQUIRE(experts >= 1 && features >= 1, "experts and features must be positive");
  PNV_REQUIRE(k > 0 && k % 8 == 0,
              "compress: K must be a multiple of 8 (whole 4-pair chunks), got %d", k);
  PNV_REQUIRE(reinterpret_cast<uintptr_t>(w_packed) % 4 == 0, "compress: the packed weights must be 4-byte aligned");
  PNV_REQUIRE((reinterpret_cast<uintptr_t>(a_comp) | reinterpret_cast<uintptr_t>(sfa)) % 16 == 0 &&
                  reinterpret_cast<uintptr_t>(e_meta) % 4 == 0,
              "compress: a_comp and sfa must be 16-byte aligned, e_meta 4-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  WeightDims wd = weight_dims(features, k);
  const long long tiles = (long long)experts * (wd.m_e / 128) * ceil_div_i(wd.k_e / 16, kTileLines);
  const long long blocks = tiles < (1LL << 30) ? tiles : (1LL << 30);
  compress_kernel<<<(unsigned)blocks, kThreads, 0, s>>>(w_packed, w_blockscale, tiles, features, k, wd, a_comp, e_meta, sfa);
  PNV_CUDA(cudaGetLastError());
  return PNV_OK;
}
