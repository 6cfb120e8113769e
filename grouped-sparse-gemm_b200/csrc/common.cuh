// Shared host/device helpers: error reporting for the C ABI, the closed-form operand layouts and
// the numeric conversions every producer shares.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/paired_nvfp4_b200.h"

namespace pnv {

// ---- error reporting -------------------------------------------------------------------------

char* last_error_buffer();   // thread-local, 512 bytes (abi.cu)

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buffer(), 512, fmt, ap);
  va_end(ap);
  return code;
}

#define PNV_REQUIRE(cond, ...)                                             \
  do {                                                                     \
    if (!(cond)) return ::pnv::fail(PNV_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
  } while (0)

#define PNV_CUDA(expr)                                                                       \
  do {                                                                                       \
    cudaError_t err__ = (expr);                                                              \
    if (err__ != cudaSuccess)                                                                \
      return ::pnv::fail(PNV_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(err__));   \
  } while (0)

// ---- layout arithmetic -------------------------------------------------------------------------
//
// Scale-factor buffers (SFA for weights, SFB for activations): one UE4M3 byte per 32 dense K
// elements, stored in 512-byte atoms of 128 rows x 4 K-blocks; K atoms innermost, then row atoms,
// then experts.  Inside an atom the scale of (row r, K-block kb) sits at byte
// (r % 32) * 16 + (r / 32 % 4) * 4 + kb % 4: 32 lines of 16 bytes, which is exactly the source
// shape of one tcgen05.cp.32x128b.warpx4 copy into tensor memory.
//
// Sparsity metadata: 4 bits per 8 dense K elements, two nibbles per byte, in atoms of
// 128 rows x 16 bytes (256 dense K), row-major inside, atoms ordered M-fastest, then K, then
// expert: the source shape of one tcgen05.cp.128x128b copy.

constexpr int kSfBlock = 32;         // dense K elements per scale
constexpr int kBenignSf = 0x38;      // UE4M3 1.0

__host__ __device__ inline int ceil_div_i(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline int round_up_i(int a, int b) { return ceil_div_i(a, b) * b; }

struct WeightDims {
  int m_ac;        // rows of a_comp
  int k_ac;        // e2m1 elements per a_comp row (bytes = k_ac / 2)
  int m_e;         // rows of e_meta
  int k_e;         // bytes per e_meta row
};

__host__ __device__ inline WeightDims weight_dims(int features, int k) {
  return WeightDims{features, round_up_i(k, 64) / 2, round_up_i(features, 128), round_up_i(k, 256) / 16};
}

__host__ __device__ inline int sf_row_atoms(int rows) { return ceil_div_i(rows, 128); }
__host__ __device__ inline int sf_k_atoms(int k) { return ceil_div_i(ceil_div_i(k, kSfBlock), 4); }
__host__ __device__ inline long long sf_numel(int rows, int k, int groups) {
  return (long long)groups * sf_row_atoms(rows) * sf_k_atoms(k) * 512;
}
// Byte offset of scale (group g, row r, K-block kb).
__host__ __device__ inline long long sf_offset(int g, int r, int kb, int n_rt, int n_kt) {
  long long atom = ((long long)g * n_rt + (r >> 7)) * n_kt + (kb >> 2);
  return atom * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4 + (kb & 3);
}

// ---- outputs spread over several buffers ---------------------------------------------------------
//
// Row q of a logical [n * rows_per_part, width] output lives at row q % rows_per_part of buffer q / rows_per_part.
// The buffers may be another GPU's memory mapped into this process (peer access): the expert-parallel exchange
// lets the producing kernel store every row straight into the buffer of the rank that wants it.
constexpr int kMaxRowParts = 16;
struct RowParts {
  void* base[kMaxRowParts];
  int n;                 // 0: a single buffer, addressed the ordinary way
  int rows_per_part;
};
inline int make_row_parts(void* const* parts, int n_parts, long long rows_per_part, RowParts& out) {
  PNV_REQUIRE(parts != nullptr, "null pointer argument");
  PNV_REQUIRE(n_parts >= 1 && n_parts <= kMaxRowParts, "between 1 and %d output parts, got %d", kMaxRowParts, n_parts);
  PNV_REQUIRE(rows_per_part >= 1 && rows_per_part < (1LL << 31), "bad rows_per_part");
  for (int i = 0; i < kMaxRowParts; ++i) out.base[i] = i < n_parts ? parts[i] : nullptr;
  for (int i = 0; i < n_parts; ++i)
    PNV_REQUIRE(parts[i] != nullptr && reinterpret_cast<uintptr_t>(parts[i]) % 16 == 0, "output part %d is null or not 16-byte aligned", i);
  out.n = n_parts;
  out.rows_per_part = (int)rows_per_part;
  return PNV_OK;
}
// Address of byte 0 of row q (rows of `pitch` bytes).
__device__ __forceinline__ uint8_t* part_row(const RowParts& parts, long long q, long long pitch) {
  const int w = (int)(q / parts.rows_per_part);
  return static_cast<uint8_t*>(parts.base[w]) + (q - (long long)w * parts.rows_per_part) * pitch;
}

// ---- programmatic dependent launch -----------------------------------------------------------

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

bool pdl_enabled();   // env PAIRED_NVFP4_PDL, read once (abi.cu)

// Launch `kernel` so that it may start before its stream predecessor has drained; the kernel
// calls pdl_wait() before its first read of anything the predecessor wrote.
template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t stream, bool pdl, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// ---- numeric conversions ------------------------------------------------------------------------

// Eight floats -> one 32-bit word of e2m1 nibbles, element j in nibble j (round-to-nearest-even, saturating to +-6).  (One
// statement: the four bytes are packed by a vector move, where separate conversions cost a widening, a shift and an or each.)
__device__ __forceinline__ uint32_t cvt_e2m1x8(const float (&v)[8]) {
  uint32_t r;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\tcvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(r) : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  return r;
}

// float -> UE4M3 byte, round-to-nearest-even, saturating to 448.
__device__ __forceinline__ uint32_t cvt_ue4m3(float x) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.0f), "f"(x));
  return (uint32_t)(r & 0xFF);
}

__device__ __forceinline__ float ue4m3_to_float(uint32_t b) {
  uint32_t h2;
  asm("{\n\t.reg .b16 t;\n\tcvt.u16.u32 t, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, t;\n\t}" : "=r"(h2) : "r"(b & 0xFFu));
  __half lo = __ushort_as_half((unsigned short)(h2 & 0xFFFF));
  return __half2float(lo);
}

// The block-scale step every quantizer shares: from the block's amax and the expert's global
// scale g, the stored UE4M3 byte and the multiplier applied before the e2m1 rounding.
//   bsf = amax > 0 ? amax / 6 : 1;  sf = ue4m3(bsf * g);  inv = float(sf) > 0 ? g / float(sf) : 0
__device__ __forceinline__ void block_scale(float amax, float g, uint32_t& sf_byte, float& inv) {
  float bsf = amax > 0.f ? __fdiv_rn(amax, 6.f) : 1.f;
  sf_byte = cvt_ue4m3(__fmul_rn(bsf, g));
  float sf = ue4m3_to_float(sf_byte);
  inv = sf > 0.f ? __fdiv_rn(g, sf) : 0.f;
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Eight bf16 (one 128-bit word) -> floats.
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  f[0] = bf16_lo(v.x); f[1] = bf16_hi(v.x); f[2] = bf16_lo(v.y); f[3] = bf16_hi(v.y);
  f[4] = bf16_lo(v.z); f[5] = bf16_hi(v.z); f[6] = bf16_lo(v.w); f[7] = bf16_hi(v.w);
}

// The gated activation applied between the two expert GEMMs, with the rounding chain of the
// unfused path: silu  -> bf16(float(bf16(g / (1 + expf(-g)))) * u)
//               situ  -> bf16((0.5 b) tanhf(g / b) (1 + tanhf(g / 2)) * (l > 0 ? l tanhf(u / l) : u))
struct GatedAct {
  int kind;
  float beta;
  float linear_beta;
  float inv_beta, inv_linear; // 1 / beta, 1 / linear_beta
  int direct;                 // SiLU: evaluate the expression itself (testing) instead of its short form
};

__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
constexpr float kLog2e = 1.44269504088896341f;

// tanh(|x|) as num / den with den = 1 + exp(-2|x|): the caller shares one reciprocal between several of them.  Above
// 0.25 num = 1 - exp(-2|x|); below, where that difference cancels, num = den * (Taylor series of tanh through x^9, whose
// next term is 1e-8 of the sum at 0.25).
__device__ __forceinline__ void tanh_parts(float x, float& num, float& den) {
  const float ax = fabsf(x);
  const float e = ex2_approx(ax * (-2.f * kLog2e));
  den = 1.f + e;
  const float x2 = ax * ax;
  const float series = fmaf(x2, fmaf(x2, fmaf(x2, fmaf(x2, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f), 1.f);
  num = ax < 0.25f ? (series * ax) * den : 1.f - e;
}

// SiTU in the form 0.5 (1 + tanh(g / 2)) = 1 / (1 + exp(-g)), everything over one common denominator: three exponentials
// and one reciprocal where the expression has three tanhf and their divisions.  For gates of unit size the result is good
// to 1e-7 before its rounding, as the expression's is; the exponent's product with log2(e) is rounded first, so the error
// grows with |g| to 5e-6 at 80, far below a bf16 unit; for negative gates, where 1 + tanhf(g / 2) cancels, the result is
// nearer to the exact one.  Not yet rounded to bf16.  (With tanhf the unfused layer of 8192 tokens on
// 128 experts of 3072 x 3072 took 1103 us, in this form 969.)
__device__ __forceinline__ float situ_short(float g, float u, float beta, float inv_beta, float linear_beta, float inv_linear) {
  float gn, gd;
  tanh_parts(__fmul_rn(g, inv_beta), gn, gd);
  float den = gd * (1.f + ex2_approx(g * -kLog2e));
  float up;
  if (linear_beta > 0.f) {
    float un, ud;
    tanh_parts(__fmul_rn(u, inv_linear), un, ud);
    den *= ud;
    up = copysignf(linear_beta * un, u);
  } else {
    up = u;
  }
  return copysignf((beta * gn) * rcp_approx(den), g) * up;
}

// bf16(g / (1 + expf(-g))) for a gate value that is itself a bf16 number.
__device__ __forceinline__ float silu_direct(float g) {
  float s = __fdiv_rn(g, __fadd_rn(1.0f, expf(-g)));
  return __bfloat162float(__float2bfloat16_rn(s));
}
// The same bits in a handful of instructions: the approximate exponential and reciprocal are good to 1e-7 for gates of unit
// size and to 5e-6 at |g| = 80 (the exponent's product is rounded), and for none of the 65536 bf16 gates does that move the
// result across a bf16 rounding boundary (checked for every pattern by the tests).  The direct form's expf and IEEE division cost about 40 instructions with a
// slow-path branch; a 65536-entry table in global memory cost one gathered load per gate, which the L1 serves at about
// 14 cycles per warp - that, not memory, was the bound of both users (gated quantizer 57 us for 12000 x 2880 outputs).
__device__ __forceinline__ float silu_short(float g) {
  const float r = rcp_approx(__fadd_rn(1.0f, ex2_approx(__fmul_rn(g, -kLog2e))));      // 1 / (1 + exp(-g))
  return __fmul_rn(g, r);
}

// General form (any activation kind).
__device__ __forceinline__ float gated_act(float g, float u, const GatedAct& a) {
  if (a.kind == PNV_ACT_SITU)
    return __bfloat162float(__float2bfloat16_rn(situ_short(g, u, a.beta, a.inv_beta, a.linear_beta, a.inv_linear)));
  const float s_bf = a.direct ? silu_direct(g) : __bfloat162float(__float2bfloat16_rn(silu_short(g)));
  return __bfloat162float(__float2bfloat16_rn(__fmul_rn(s_bf, u)));
}

// ---- two bf16 to a register ----------------------------------------------------------------------
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// Element-wise max of two pairs of magnitudes (a NaN loses to a number, as with fmaxf).
__device__ __forceinline__ uint32_t bf16x2_max(uint32_t a, uint32_t b) { return as_u32(__hmax2(as_bf162(a), as_bf162(b))); }
// Largest magnitude of eight pairs, separately for the low and the high halves.
__device__ __forceinline__ uint32_t bf16x2_amax8(const uint32_t (&y)[8]) {
  uint32_t m = y[0] & 0x7FFF7FFFu;
#pragma unroll
  for (int i = 1; i < 8; ++i) m = bf16x2_max(m, y[i] & 0x7FFF7FFFu);
  return m;
}
// Eight bf16 in four registers -> one word of e2m1 codes after scaling by inv (two products to an instruction, each rounded
// as on its own).
__device__ __forceinline__ uint32_t quant8_packed(uint32_t a, uint32_t b, uint32_t c, uint32_t d, float inv) {
  const uint32_t w[4] = {a, b, c, d};
  float v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(v[2 * i]), "=f"(v[2 * i + 1]) : "f"(bf16_lo(w[i])), "f"(bf16_hi(w[i])), "f"(inv));
  return cvt_e2m1x8(v);
}
// The gated activation of 16 neighbouring features.  silu(g) is a bf16 number and the product of two bf16 numbers is
// exact in float, so one packed bf16 multiplication rounds like the float product rounded to bf16.
__device__ __forceinline__ void gated_act16(const uint32_t (&g)[8], const uint32_t (&u)[8], const GatedAct& a, uint32_t (&y)[8]) {
  if (a.kind == PNV_ACT_SILU && !a.direct) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_bfloat162 s = __floats2bfloat162_rn(silu_short(bf16_lo(g[i])), silu_short(bf16_hi(g[i])));
      y[i] = as_u32(__hmul2(s, as_bf162(u[i])));
    }
  } else if (a.kind == PNV_ACT_SITU) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      y[i] = as_u32(__floats2bfloat162_rn(situ_short(bf16_lo(g[i]), bf16_lo(u[i]), a.beta, a.inv_beta, a.linear_beta, a.inv_linear),
                                          situ_short(bf16_hi(g[i]), bf16_hi(u[i]), a.beta, a.inv_beta, a.linear_beta, a.inv_linear)));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      y[i] = as_u32(__floats2bfloat162_rn(gated_act(bf16_lo(g[i]), bf16_lo(u[i]), a), gated_act(bf16_hi(g[i]), bf16_hi(u[i]), a)));
  }
}

// (activation kind, beta, linear_beta) -> GatedAct with the reference's argument checks (quant.cu)
int make_gated_act(int act_kind, float beta, float linear_beta, GatedAct& out);

}  // namespace pnv
