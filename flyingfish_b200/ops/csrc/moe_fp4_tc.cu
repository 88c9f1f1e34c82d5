// Grouped expert GEMM over NVFP4 weights for batches of 16 and more rows an expert on average, on tcgen05 (formats, rounding and epilogues as in
// moe_fp4.cu, which serves segments of a few rows; prompts of more than 32 rows an expert take the BF16 copies that the layer keeps):
//   Y[seg rows, Nw] = Xs[seg rows, K] · (e2m1(Wq[e]) * e4m3(Wsc[e]) * global[e])[Nw, K]ᵀ
// moe_fp4.cu expands a weight tile once for every 32 rows of a segment, which is what its time goes by; here it is expanded once for up to 256.
// Whole expert layer (128 experts of 4096 x 1536), us with moe_fp4.cu / here: 8 rows an expert 540 / 738, 12.5 652 / 740, 16 757 / 742, 32
// 1241 / 759; on BF16 copies of the experts 752, 846, 845 and 878. The packed bytes take 207.
//   * Persistent CTAs, one per SM, walk the (expert, 128 weight rows) tiles of the experts that have rows; a pass multiplies up to 256 rows.
//     The weights are the 128-row operand A, the rows the N dimension: a weight tile is expanded once for all rows of a pass.
//   * Roles: a warp that copies packed chunks (256 of K: codes and scales), one that copies the rows' K blocks, one that multiplies, sixteen that
//     expand a 64-wide K block of A (128-byte swizzled, K-major) from a chunk, four that write finished tiles. Three stages between each two.
//   * Expanding takes a word of eight codes 17 instructions and four permutes, about 300 cycles of the four schedulers for a K block, which takes the
//     tensor cores 288 cycles with 144 rows; a K block takes about 650 cycles, with eight warps 680: shared memory (about 480 cycles of reads and writes) and
//     the fences between the expanding warps' writes and the tensor cores.
// Every wait is bounded; warps that share a named barrier leave a failed pass together.
#include "ptx.cuh"
#include "host_util.h"
#include "fp4_expand.cuh"

namespace ff {

constexpr int FT_M = 128, FT_KC = 256, FT_KB = 64, FT_TOK = 256;
constexpr int FT_CODES = FT_M * FT_KC / 2, FT_SCALES = FT_M * FT_KC / 16, FT_CHUNK = FT_CODES + FT_SCALES;      // 18 KiB
constexpr int FT_A = FT_M * FT_KB * 2, FT_B = FT_TOK * FT_KB * 2, FT_BOX = 64;                                   // 16 and 32 KiB
constexpr int FT_STAGES = 3, FT_PITCH = FT_M + 4, FT_OUT = 32 * FT_PITCH * 4;
constexpr int FT_SMEM = FT_STAGES * (FT_A + FT_B + FT_CHUNK) + FT_OUT + 1024;                                    // 217 KiB, and the list of experts
constexpr int FT_EXPAND = 16, FT_THREADS = 32 * (3 + FT_EXPAND + 4);

struct alignas(8) Fp4TcBars {
  uint64_t p_full[FT_STAGES], p_empty[FT_STAGES], a_full[FT_STAGES], a_empty[FT_STAGES], b_full[FT_STAGES], b_empty[FT_STAGES];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag, active;
};

__device__ __forceinline__ float ft_silu(float x) { return x / (1.0f + __expf(-x)); }
__device__ __forceinline__ float ft_bfr(float x) { return __bfloat162float(__float2bfloat16(x)); }
// barrier of the four writing warps, and whether any of them passed true
__device__ __forceinline__ bool ft_sync_any(bool mine) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((uint32_t)mine) : "memory");
  return any != 0;
}

__global__ void __launch_bounds__(FT_THREADS, 1)
moe_fp4_tc_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS, const __grid_constant__ CUtensorMap tmX,
                  const float* __restrict__ Wglobal, __nv_bfloat16* __restrict__ Y, const int* __restrict__ seg_off, const int* __restrict__ counts, int E,
                  int Nw, int K, int ldy, int epi, int capacity, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Fp4TcBars bars;
  uint8_t* sA = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sB = sA + FT_STAGES * FT_A;
  uint8_t* sP = sB + FT_STAGES * FT_B;
  float* sT = reinterpret_cast<float*>(sP + FT_STAGES * FT_CHUNK);           // 32 rows of a finished tile
  int3* act = reinterpret_cast<int3*>(reinterpret_cast<uint8_t*>(sT) + FT_OUT);   // experts with rows: id, first row, rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmS); tma_prefetch_desc(&tmX);
    for (int i = 0; i < FT_STAGES; ++i) {
      mbar_init(&bars.p_full[i], 1); mbar_init(&bars.p_empty[i], FT_EXPAND);
      mbar_init(&bars.a_full[i], FT_EXPAND); mbar_init(&bars.a_empty[i], 1);
      mbar_init(&bars.b_full[i], 1); mbar_init(&bars.b_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) { mbar_init(&bars.tmem_full[i], 1); mbar_init(&bars.tmem_empty[i], 4); }
    bars.abort_flag = 0;
    mbar_fence_init();
  }
  pdl_wait();                                              // rows, offsets and counts are the preceding kernels'
  if (warp == 1) { tmem_alloc(&bars.tmem_base, 512); tmem_relinquish(); }
  if (warp == 2) {
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
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  const uint32_t tmem_base = bars.tmem_base;
  volatile int* abort_flag = &bars.abort_flag;
  const int tiles_n = Nw / FT_M, items = bars.active * tiles_n, chunks = K / FT_KC, kblocks = K / FT_KB;
  // every role walks the same passes: rows p .. p + 255 of the segment of item w
  auto pass_rows = [&](int left) { return min(FT_TOK, left); };

  if (warp == 0) {                                          // packed chunks
    if (elect_one()) {
      const uint64_t pol = l2_policy_evict_first();
      RingPos rp;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int3 a = act[w / tiles_n];
        const int wrow = a.x * Nw + (w % tiles_n) * FT_M;
        for (int p = 0; p < a.z && ok; p += FT_TOK)
          for (int c = 0; c < chunks; ++c, rp.next(FT_STAGES)) {
            if (!mbar_wait(&bars.p_empty[rp.s], rp.ph ^ 1, abort_flag, status, KID_MOE_GEMM, 21)) { ok = false; break; }
            mbar_expect_tx(&bars.p_full[rp.s], FT_CHUNK);
            tma_load_2d_hint(sP + rp.s * FT_CHUNK, &tmW, &bars.p_full[rp.s], c * (FT_KC / 2), wrow, pol);
            tma_load_2d(sP + rp.s * FT_CHUNK + FT_CODES, &tmS, &bars.p_full[rp.s], c * (FT_KC / 16), wrow);
          }
      }
    }
  } else if (warp == 2) {                                   // rows
    if (elect_one()) {
      RingPos rp;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int3 a = act[w / tiles_n];
        for (int p = 0; p < a.z && ok; p += FT_TOK) {
          // whole boxes of 64 rows: what lies behind the segment is read and not multiplied
          const int boxes = (pass_rows(a.z - p) + FT_BOX - 1) / FT_BOX;
          for (int kb = 0; kb < kblocks; ++kb, rp.next(FT_STAGES)) {
            if (!mbar_wait(&bars.b_empty[rp.s], rp.ph ^ 1, abort_flag, status, KID_MOE_GEMM, 22)) { ok = false; break; }
            mbar_expect_tx(&bars.b_full[rp.s], boxes * FT_BOX * FT_KB * 2);
            for (int i = 0; i < boxes; ++i)
              tma_load_2d(sB + rp.s * FT_B + i * FT_BOX * FT_KB * 2, &tmX, &bars.b_full[rp.s], kb * FT_KB, a.y + p + i * FT_BOX);
          }
        }
      }
    }
  } else if (warp == 1) {                                   // products
    if (elect_one()) {
      RingPos rp;
      uint32_t pass_it = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int3 a = act[w / tiles_n];
        for (int p = 0; p < a.z && ok; p += FT_TOK, ++pass_it) {
          const uint32_t idesc = umma_idesc(1, 1, 0, 0, FT_M, (pass_rows(a.z - p) + 15) / 16 * 16);
          const int acc = pass_it & 1;
          if (!mbar_wait(&bars.tmem_empty[acc], ((pass_it >> 1) & 1) ^ 1, abort_flag, status, KID_MOE_GEMM, 23)) { ok = false; break; }
          tc_fence_after();
          for (int kb = 0; kb < kblocks; ++kb, rp.next(FT_STAGES)) {
            const int s = rp.s;
            if (!mbar_wait(&bars.b_full[s], rp.ph, abort_flag, status, KID_MOE_GEMM, 24) ||
                !mbar_wait(&bars.a_full[s], rp.ph, abort_flag, status, KID_MOE_GEMM, 25)) { ok = false; break; }
            tc_fence_after();
            const uint64_t da = umma_desc_sw128(smem_u32(sA + s * FT_A), 16, 1024), db = umma_desc_sw128(smem_u32(sB + s * FT_B), 16, 1024);
#pragma unroll
            for (int k = 0; k < FT_KB / 16; ++k) umma_f16(tmem_base + acc * FT_TOK, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
            umma_commit(&bars.a_empty[s]);
            umma_commit(&bars.b_empty[s]);
          }
          if (ok) umma_commit(&bars.tmem_full[acc]);
        }
      }
    }
  } else if (warp < 3 + FT_EXPAND) {                        // expanding: thread -> weight row, 16 of a K block's 64 columns (one scale)
    const int tid = threadIdx.x - 96, row = tid & 127, part = tid >> 7, sw = row & 7;
    RingPos pp, ap;
    bool ok = true;
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const int rows = act[w / tiles_n].z;
      for (int p = 0; p < rows && ok; p += FT_TOK)
        for (int c = 0; c < chunks && ok; ++c, pp.next(FT_STAGES)) {
          if (!__all_sync(0xffffffffu, mbar_wait(&bars.p_full[pp.s], pp.ph, abort_flag, status, KID_MOE_GEMM, 26))) { ok = false; break; }
          const uint8_t* st = sP + pp.s * FT_CHUNK;
          uint2 q[4];
          uint32_t sc[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            q[j] = *reinterpret_cast<const uint2*>(st + row * 128 + (((2 * j + (part >> 1)) ^ sw) << 4) + (part & 1) * 8);
            sc[j] = st[FT_CODES + row * 16 + j * 4 + part];
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            __nv_bfloat162 s2, unused;
            f4_scale2(sc[j], s2, unused);
            const uint32_t words[2] = {q[j].x, q[j].y};
            uint4 o[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              uint32_t v[4];                                // pairs (0, 4), (1, 5), (2, 6), (3, 7)
              f4_expand8(words[i], s2, v);
              o[i] = make_uint4(__byte_perm(v[0], v[1], 0x5410), __byte_perm(v[2], v[3], 0x5410), __byte_perm(v[0], v[1], 0x7632), __byte_perm(v[2], v[3], 0x7632));
            }
            if (ok && !__all_sync(0xffffffffu, mbar_wait(&bars.a_empty[ap.s], ap.ph ^ 1, abort_flag, status, KID_MOE_GEMM, 27))) ok = false;
            if (!ok) break;
            uint8_t* dst = sA + ap.s * FT_A + row * 128;
#pragma unroll
            for (int i = 0; i < 2; ++i) *reinterpret_cast<uint4*>(dst + (((part * 2 + i) ^ sw) << 4)) = o[i];
            fence_proxy_async_smem();                       // read by the tensor cores
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.a_full[ap.s]);
            ap.next(FT_STAGES);
          }
          // The chunk is given back behind the stores that its codes went into. An arrival right behind the loads does not wait for them: where the tensor
          // cores held the expanding warps up (segments from about 150 rows) the refill overtook the loads of the chunk's last K blocks.
          if (ok && lane == 0) mbar_arrive(&bars.p_empty[pp.s]);
        }
    }
  } else {                                                  // finished tiles: lane = weight row, columns = rows of the segment
    const int q = warp & 3, nl = q * 32 + lane, ee = threadIdx.x - 32 * (3 + FT_EXPAND);
    uint32_t pass_it = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const int3 a = act[w / tiles_n];
      const int tn = w % tiles_n;
      const float gscale = Wglobal[a.x] * 256.0f;
      for (int p = 0; p < a.z && ok; p += FT_TOK, ++pass_it) {
        const int acc = pass_it & 1, real = pass_rows(a.z - p);
        const bool got = mbar_wait(&bars.tmem_full[acc], (pass_it >> 1) & 1, abort_flag, status, KID_MOE_GEMM, 28);
        if (ft_sync_any(!got)) { ok = false; break; }       // also: the staging rows of the last pass have been read
        tc_fence_after();
        const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + acc * FT_TOK;
        for (int t0 = 0; t0 < real; t0 += 32) {
          uint32_t r[32];
          tmem_ld_x32(taddr + t0, r);
          tmem_ld_wait();
          if (t0) asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j) sT[j * FT_PITCH + nl] = __uint_as_float(r[j]) * gscale;
          asm volatile("bar.sync 1, 128;" ::: "memory");
          const int n = min(32, real - t0);
          __nv_bfloat16* y0 = Y + (size_t)(a.y + p + t0) * ldy;
          if (epi == 1) {
            const int c8 = ee & 7;
            for (int t = ee >> 3; t < n; t += 16) {
              const float* g = sT + t * FT_PITCH + c8 * 8;
              uint32_t o[4];
#pragma unroll
              for (int j = 0; j < 4; ++j)
                o[j] = pack_bf16x2(ft_bfr(ft_silu(ft_bfr(g[2 * j]))) * ft_bfr(g[64 + 2 * j]), ft_bfr(ft_silu(ft_bfr(g[2 * j + 1]))) * ft_bfr(g[64 + 2 * j + 1]));
              *reinterpret_cast<uint4*>(y0 + (size_t)t * ldy + tn * 64 + c8 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
            }
          } else {
            const int c16 = ee & 15;
            for (int t = ee >> 4; t < n; t += 8) {
              const float* g = sT + t * FT_PITCH + c16 * 8;
              uint32_t o[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(g[2 * j], g[2 * j + 1]);
              *reinterpret_cast<uint4*>(y0 + (size_t)t * ldy + tn * FT_M + c16 * 8) = make_uint4(o[0], o[1], o[2], o[3]);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.tmem_empty[acc]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (bars.abort_flag) {                                    // copies still in flight land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
  }
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

}  // namespace ff
using namespace ff;

// The operands of ff_moe_grouped_gemm_nvfp4 (moe_fp4.cu); K a multiple of 256.
FF_EXPORT int ff_moe_grouped_gemm_nvfp4_tc(const void* xs, const void* wq, const void* wsc, const float* wglobal, void* y, const int* seg_off,
                                           const int* counts, int E_local, int Nw, int K, int capacity, int ldy, int epi, int* status, cudaStream_t s) {
  if (E_local <= 0 || E_local > 768 || Nw <= 0 || K <= 0 || capacity <= 0 || !seg_off || !counts || !wglobal) return FF_HOST_BAD_SHAPE;
  if (Nw % FT_M || K % FT_KC || (epi != 0 && epi != 1)) return FF_HOST_BAD_SHAPE;
  if (ldy % 8 || ldy < (epi == 1 ? Nw / 2 : Nw)) return FF_HOST_BAD_ALIGN;
  if ((reinterpret_cast<uintptr_t>(xs) | reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(wsc) | reinterpret_cast<uintptr_t>(y)) & 15) return FF_HOST_BAD_ALIGN;
  CUtensorMap tmW, tmS, tmX;
  const uint64_t wrows = (uint64_t)E_local * Nw;
  if (int r = make_tmap_2d(&tmW, wq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 2, wrows, K / 2, FT_KC / 2, FT_M)) return r;
  if (int r = make_tmap_2d(&tmS, wsc, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K / 16, wrows, K / 16, FT_KC / 16, FT_M, false)) return r;
  if (int r = make_tmap_2d(&tmX, xs, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, capacity, (uint64_t)K * 2, FT_KB, FT_BOX)) return r;
  const int smem = FT_SMEM + E_local * 12;
  if (int r = opt_in_smem(moe_fp4_tc_kernel, FT_SMEM + 768 * 12)) return r;
  const long long tiles = (long long)E_local * (Nw / FT_M);
  const int grid = tiles < sm_count() ? (int)tiles : sm_count();
  return launch_pdl(moe_fp4_tc_kernel, dim3(grid), dim3(FT_THREADS), smem, s, 0, tmW, tmS, tmX, wglobal, (__nv_bfloat16*)y, seg_off, counts, E_local, Nw, K, ldy, epi,
                    capacity, status);
}
