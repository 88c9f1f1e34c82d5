// Grouped expert GEMM over NVFP4 weights without a BF16 copy of them in memory (W4A16):
//   Y[seg rows, Nw] = Xs[seg rows, K] · (e2m1(Wq[e]) * e4m3(Wsc[e]) * global[e])[Nw, K]ᵀ
// Wq  : [E_local * Nw, K / 2] bytes, two E2M1 codes per byte, low nibble first
// Wsc : [E_local * Nw, K / 16] bytes, one E4M3 scale per 16 weights
// global : FP32 per expert (ModelOpt `weight_scale_2`)
// The decode-sized MoE layer is bound by expert weight bytes, so the weights stay packed in HBM (a quarter of the
// BF16 bytes) and are expanded in the registers of the warps that multiply them (mma.sync, weights as the 16-row A fragment, tokens
// as the 8 columns of B). Why not tcgen05: with converters in front of its 128-row operand the one thread that waits for, issues and
// commits four products per 64-wide block held a GPU at 1.7 TB/s of packed bytes, with the expansion left out and through shared or
// tensor memory alike (528 us for a gate/up product of 0.9 GB); here every warp multiplies what it has just expanded.
//   * Persistent CTAs, two per SM, walk the (expert, 128 weight rows) tiles of the experts that have tokens. A producer warp keeps a ring
//     of 256-wide K chunks (codes and scales) in flight with TMA; lanes that read 64-byte pieces of eight rows from global memory
//     themselves reached 2.9 TB/s with nothing else to do. Eight warps own 16 weight rows each: lane (g, t) takes 16 bytes (32 codes)
//     of rows g and g + 8 at a time. The codes of a word go to the K slots of two mma in the order in which expanding leaves them;
//     the tokens are put into shared memory in that order once per slab, as conflict-free 16-byte units.
//   * Expanding: the three magnitude bits of a code moved to bits 8..6 of a BF16 are the value times 2^-126 (the subnormal 0.5
//     included); one BF16x2 multiply by the group's scale times 2^118 makes it e2m1 * e4m3 * 2^-8, exactly (2 + 4 significant
//     bits). The 2^8 goes with the per-expert global scale, which is applied in FP32 in the epilogue, with the optional SwiGLU of
//     gate/up stacks interleaved per 64 rows.
//   * Up to 32 tokens per pass (1, 2 or 4 column tiles; the tokens of 512 to 2048 K at a time in 32 KB). Longer segments take
//     passes that expand again, so this kernel is meant for decode-sized segments; prefill-sized calls use the tiled grouped GEMM
//     over BF16 weights.
// 128 experts of 4096 x 1536 with 2 rows each: gate/up and down 658 + 342 us with converters in front of tcgen05, 290 + 154 us now (packed
// bytes at the copy rate: 138 + 69 us); what is left is integer work, 0.65 of the issue slots busy.
// Format: kernels/nvfp4_linear.cu and src/fp8.rs:124-147 of the reference.
#include "ptx.cuh"
#include "host_util.h"
#include "pass_walk.h"
#include "fp4_expand.cuh"
#include <type_traits>

namespace ff {

constexpr int F4_BM = 128;           // weight rows per CTA
constexpr int F4_KC = 256;           // K of a ring stage: 128 bytes of codes and 16 scales per row
constexpr int F4_TOK = 32;           // most tokens per pass
constexpr int F4_WARPS = 8;          // multiplying warps, 16 weight rows each; one more produces
constexpr int F4_THREADS = 32 * F4_WARPS + 32;
constexpr int F4_CODES = F4_BM * F4_KC / 2, F4_SCALES = F4_BM * F4_KC / 16, F4_STAGE = F4_CODES + F4_SCALES;      // 18 KiB
constexpr int F4_STAGES = 3;
constexpr int F4_X_BYTES = 32 * 1024;                // tokens of a K slab: 8 * NT of them, 2048 / NT wide; then the epilogue's FP32 tile

struct alignas(8) Fp4Bars {
  uint64_t full[F4_STAGES];
  uint64_t empty[F4_STAGES];
  int abort_flag;
  int active;
};
__device__ __forceinline__ void f4_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }      // the multiplying warps
// the same, and whether any of them passed true
__device__ __forceinline__ bool f4_sync_any(bool mine) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((uint32_t)mine) : "memory");
  return any != 0;
}

__device__ __forceinline__ float f4_silu(float x) { return x / (1.0f + __expf(-x)); }
__device__ __forceinline__ float f4_bfr(float x) { return __bfloat162float(__float2bfloat16(x)); }

__device__ __forceinline__ void f4_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One pass: `real` (at most 8 NT) tokens from row `grow0` of X against the 128 weight rows that come through the ring. `it`: stages used so far.
template <int NT>
__device__ __forceinline__ bool f4_pass(const __nv_bfloat16* __restrict__ X, int grow0, int real, uint8_t* ring, Fp4Bars& bars, uint32_t& it,
                                        const uint8_t* __restrict__ wsc, int K, uint8_t* xbuf, float gscale, __nv_bfloat16* __restrict__ Y,
                                        int ldy, int tn, int epi, int* status) {
  constexpr int SLAB = F4_X_BYTES / (16 * NT);         // K that the tokens in shared memory cover
  static_assert(SLAB % F4_KC == 0, "a slab holds whole stages");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int chunks = (K + F4_KC - 1) / F4_KC, ra = warp * 16 + g;       // rows ra and ra + 8 have the same swizzle
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

  constexpr int PER_SLAB = SLAB / F4_KC;
  auto fill = [&](int c) {
    // tokens of this slab: unit [128-wide K][column tile][i2][token][t] holds x[token][32 t + 8 i2 + {0,4,1,5,2,6,3,7}]
    const int k0 = c * F4_KC, per = min(SLAB, K - k0) / 8;
    for (int i = threadIdx.x; i < 8 * NT * per; i += 32 * F4_WARPS) {
      const int n = i / per, k8 = i - n * per;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (n < real) v = __ldg(reinterpret_cast<const uint4*>(X + (size_t)(grow0 + n) * K + k0) + k8);
      const int ch = k8 >> 4, tt = (k8 >> 2) & 3, i2 = k8 & 3;
      *reinterpret_cast<uint4*>(xbuf + ((((ch * NT + (n >> 3)) * 4 + i2) * 8 + (n & 7)) * 4 + tt) * 16) =
          make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632), __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
    }
  };
  auto wait = [&](int) {
    return __all_sync(0xffffffffu, mbar_wait(&bars.full[it % F4_STAGES], (it / F4_STAGES) & 1, &bars.abort_flag, status, KID_MOE_GEMM, 15)) != 0;
  };
  auto multiply = [&](int c) {
    const int in_slab = c % PER_SLAB, s = it % F4_STAGES;
    ++it;
    const uint8_t* st = ring + s * F4_STAGE;
    uint4 qa[2], qb[2];
    uint32_t sa[2], sb[2];
    const int halves = (K - c * F4_KC) >= F4_KC ? 2 : 1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int piece = ((h * 4 + t) ^ (ra & 7)) << 4;
      qa[h] = *reinterpret_cast<const uint4*>(st + ra * 128 + piece);
      qb[h] = *reinterpret_cast<const uint4*>(st + (ra + 8) * 128 + piece);
      if (wsc == nullptr) {
        sa[h] = *reinterpret_cast<const unsigned short*>(st + F4_CODES + ra * 16 + h * 8 + t * 2);
        sb[h] = *reinterpret_cast<const unsigned short*>(st + F4_CODES + (ra + 8) * 16 + h * 8 + t * 2);
      } else {                                            // rows of scales that are no whole 16 bytes
        const uint8_t* p = wsc + (size_t)ra * (K / 16) + c * 16 + h * 8 + t * 2;
        sa[h] = h < halves ? __ldg(reinterpret_cast<const unsigned short*>(p)) : 0;
        sb[h] = h < halves ? __ldg(reinterpret_cast<const unsigned short*>(p + (size_t)8 * (K / 16))) : 0;
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h < halves) {
        const uint8_t* xs = xbuf + (size_t)(in_slab * 2 + h) * NT * 2048 + lane * 16;
        __nv_bfloat162 ga[2], gb[2];
        f4_scale2(sa[h], ga[0], ga[1]);
        f4_scale2(sb[h], gb[0], gb[1]);
        const uint32_t wa[4] = {qa[h].x, qa[h].y, qa[h].z, qa[h].w}, wb[4] = {qb[h].x, qb[h].y, qb[h].z, qb[h].w};
#pragma unroll
        for (int i2 = 0; i2 < 4; ++i2) {
          uint32_t pa[4], pb[4];
          f4_expand8(wa[i2], ga[i2 >> 1], pa);
          f4_expand8(wb[i2], gb[i2 >> 1], pb);
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const uint4 x = *reinterpret_cast<const uint4*>(xs + (j * 4 + i2) * 512);
            f4_mma(acc[j], pa[0], pb[0], pa[1], pb[1], x.x, x.y);
            f4_mma(acc[j], pa[2], pb[2], pa[3], pb[3], x.z, x.w);
          }
        }
      }
    }
    // The stage is given back behind its last multiplication, and the arrival's address goes through that sum (epi is 0 or 1): an arrival does not wait
    // for loads in front of it, and right behind them a refill could overtake those that have not returned.
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.empty[s + (__float_as_uint(acc[0][0]) & ((uint32_t)epi >> 1))]);
  };
  if (!walk_pass(chunks, PER_SLAB, f4_sync, fill, wait, multiply, f4_sync_any)) return false;
  // ---- epilogue through an FP32 transpose tile [token][128] in the tokens' place
  float* sT = reinterpret_cast<float*>(xbuf);
  const int r = ra, t2 = t * 2;
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    sT[(j * 8 + t2) * F4_BM + r] = acc[j][0] * gscale;
    sT[(j * 8 + t2 + 1) * F4_BM + r] = acc[j][1] * gscale;
    sT[(j * 8 + t2) * F4_BM + r + 8] = acc[j][2] * gscale;
    sT[(j * 8 + t2 + 1) * F4_BM + r + 8] = acc[j][3] * gscale;
  }
  f4_sync();
  if (epi == 1) {
    const int c8 = threadIdx.x & 7;                                     // 32 token rows per sweep, 8 outputs per thread
    for (int n = threadIdx.x >> 3; n < real; n += 4 * F4_WARPS) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int col = c8 * 8 + 2 * j;
        const float g0 = f4_bfr(sT[n * F4_BM + col]), g1 = f4_bfr(sT[n * F4_BM + col + 1]);
        const float u0 = f4_bfr(sT[n * F4_BM + 64 + col]), u1 = f4_bfr(sT[n * F4_BM + 64 + col + 1]);
        o[j] = pack_bf16x2(f4_bfr(f4_silu(g0)) * u0, f4_bfr(f4_silu(g1)) * u1);
      }
      *reinterpret_cast<uint4*>(Y + (size_t)(grow0 + n) * ldy + tn * 64 + c8 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  } else {
    const int c16 = threadIdx.x & 15;                                   // 16 token rows per sweep
    for (int n = threadIdx.x >> 4; n < real; n += 2 * F4_WARPS) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(sT[n * F4_BM + c16 * 8 + 2 * j], sT[n * F4_BM + c16 * 8 + 2 * j + 1]);
      *reinterpret_cast<uint4*>(Y + (size_t)(grow0 + n) * ldy + tn * F4_BM + c16 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  return true;
}

// persistent, two CTAs per SM; scale_tma: the scales' rows are multiples of 16 bytes and come with the ring, otherwise the lanes read them
__global__ void __launch_bounds__(F4_THREADS, 2)
moe_fp4_grouped_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS, const __nv_bfloat16* __restrict__ X,
                       const uint8_t* __restrict__ Wsc, const float* __restrict__ Wglobal, __nv_bfloat16* __restrict__ Y,
                       const int* __restrict__ seg_off, const int* __restrict__ counts, int E, int Nw, int K, int ldy, int epi, int scale_tma,
                       int capacity, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Fp4Bars bars;
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* xbuf = ring + F4_STAGES * F4_STAGE;
  int3* act = reinterpret_cast<int3*>(xbuf + F4_X_BYTES);                // experts with tokens: id, first row, rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmS);
    for (int i = 0; i < F4_STAGES; ++i) { mbar_init(&bars.full[i], 1); mbar_init(&bars.empty[i], F4_WARPS); }
    bars.abort_flag = 0;
    mbar_fence_init();
  }
  pdl_trigger();
  pdl_wait();                                             // tokens, offsets and counts are the preceding kernels'
  if (warp == 1) {
    int n = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, off = e < E ? seg_off[e] : 0;
      // a segment reaching past the row buffers (an overflowed dispatch, reported through the status word) is cut there
      const int cnt = e < E ? min(counts[e], capacity - off) : 0;
      const uint32_t m = __ballot_sync(0xffffffffu, cnt > 0);
      if (cnt > 0) act[n + __popc(m & ((1u << lane) - 1))] = make_int3(e, off, cnt);
      n += __popc(m);
    }
    if (lane == 0) bars.active = n;
  }
  __syncthreads();
  const int tiles_n = Nw / F4_BM, items = bars.active * tiles_n, chunks = (K + F4_KC - 1) / F4_KC;
  uint32_t it = 0;
  bool ok = true;
  if (warp == F4_WARPS) {
    if (lane == 0) {
      const uint64_t pol = l2_policy_evict_first();
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int3 a = act[w / tiles_n];
        const int wrow = a.x * Nw + (w % tiles_n) * F4_BM;
        for (int p = 0; p < a.z && ok; p += F4_TOK)
          for (int c = 0; c < chunks; ++c, ++it) {
            const int s = it % F4_STAGES;
            if (!mbar_wait(&bars.empty[s], ((it / F4_STAGES) & 1) ^ 1, &bars.abort_flag, status, KID_MOE_GEMM, 11)) { ok = false; break; }
            mbar_expect_tx(&bars.full[s], F4_CODES + (scale_tma ? F4_SCALES : 0));
            tma_load_2d_hint(ring + s * F4_STAGE, &tmW, &bars.full[s], c * (F4_KC / 2), wrow, pol);
            if (scale_tma) tma_load_2d(ring + s * F4_STAGE + F4_CODES, &tmS, &bars.full[s], c * (F4_KC / 16), wrow);
          }
      }
    }
  } else {
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const int3 a = act[w / tiles_n];
      const int tn = w % tiles_n;
      const uint8_t* wsc = scale_tma ? nullptr : Wsc + ((size_t)a.x * Nw + (size_t)tn * F4_BM) * (K / 16);
      const float gscale = Wglobal[a.x] * 256.0f;
      for (int p = 0; p < a.z && ok; p += F4_TOK) {
        const int real = min(F4_TOK, a.z - p);
        auto pass = [&](auto nt) {
          return f4_pass<decltype(nt)::value>(X, a.y + p, real, ring, bars, it, wsc, K, xbuf, gscale, Y, ldy, tn, epi, status);
        };
        ok = real <= 8 ? pass(std::integral_constant<int, 1>{}) : real <= 16 ? pass(std::integral_constant<int, 2>{}) : pass(std::integral_constant<int, 4>{});
      }
    }
  }
  if (!ok) {                                              // a wait ran out: copies still in flight land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
  }
}

}  // namespace ff
using namespace ff;

// Xs [capacity, K] bf16 sorted token rows; Wq / Wsc / Wglobal as described at the top; Y [capacity, ldy] bf16.
// epi 0: Y has Nw columns; epi 1: SwiGLU of gate/up rows interleaved per 64, Y has Nw / 2 columns.
FF_EXPORT int ff_moe_grouped_gemm_nvfp4(const void* xs, const void* wq, const void* wsc, const float* wglobal, void* y,
                                        const int* seg_off, const int* counts, int E_local, int Nw, int K, int capacity,
                                        int ldy, int epi, int* status, cudaStream_t s) {
  if (E_local <= 0 || Nw <= 0 || K <= 0 || capacity <= 0 || !seg_off || !counts || !wglobal) return FF_HOST_BAD_SHAPE;
  if (Nw % F4_BM || K % 128 || (epi != 0 && epi != 1)) return FF_HOST_BAD_SHAPE;
  if (ldy % 8 || ldy < (epi == 1 ? Nw / 2 : Nw)) return FF_HOST_BAD_ALIGN;
  if ((reinterpret_cast<uintptr_t>(xs) & 15) || (reinterpret_cast<uintptr_t>(wq) & 15) || (reinterpret_cast<uintptr_t>(wsc) & 15) ||
      (reinterpret_cast<uintptr_t>(y) & 15)) return FF_HOST_BAD_ALIGN;
  CUtensorMap tmW, tmS;
  const uint64_t wrows = (uint64_t)E_local * Nw;
  int r = make_tmap_2d(&tmW, wq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 2, wrows, K / 2, F4_KC / 2, F4_BM);
  if (r) return r;
  const int scale_tma = K % 256 == 0;                  // a map needs rows of whole 16 bytes
  tmS = tmW;
  if (scale_tma) { r = make_tmap_2d(&tmS, wsc, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 16, wrows, K / 16, F4_KC / 16, F4_BM, false); if (r) return r; }
  const int smem = F4_STAGES * F4_STAGE + F4_X_BYTES + E_local * 12 + 1024;
  r = opt_in_smem(moe_fp4_grouped_kernel, smem); if (r) return r;
  const long long tiles = (long long)E_local * (Nw / F4_BM);
  const int grid = tiles < 2 * sm_count() ? (int)tiles : 2 * sm_count();
  if (int lr_ = launch_pdl(moe_fp4_grouped_kernel, dim3(grid), dim3(F4_THREADS), smem, s, 0, tmW, tmS, (const __nv_bfloat16*)xs, (const uint8_t*)wsc,
                           wglobal, (__nv_bfloat16*)y, seg_off, counts, E_local, Nw, K, ldy, epi, scale_tma, capacity, status)) return lr_;
  return launch_result();
}
