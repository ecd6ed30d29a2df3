// Block-scaled fp8 grouped GEMM for few rows per expert.  As in narrow_gemm.cu the weights are the 128-row operand of the
// tensor core (a tile is two 128-row blocks) and up to 128 token rows its N columns, so that what the ring keeps in flight
// are weight bytes.  The first GEMM pairs the gate and the up block of 128 features and finishes the activation in its
// epilogue: a tile holds all 128 features of a token's scale block, so SwiGLU and the 1 x 128 quantisation need no
// second pass over the rows (and the pre-activations never reach memory).
//
// One accumulator buffer (two blocks of 128 columns): the epilogue reads its share into registers and hands the buffer
// back at once.  A tile streams 0.5 to 2 MB of weights, the hand-over costs about half a microsecond and the ring keeps
// loading meanwhile; the scale factors need the tensor memory that a second buffer would take.
//
// Warps: 0 TMA producer, 1 tensor memory + scale copies + MMA issue, 2-9 epilogue.  Every mbarrier wait is bounded; on a
// timeout the CTA raises its abort flag, records a status, lets issued copies land, frees its tensor memory and returns.
#include "narrow_gemm_fp8.h"

#include <cuda_bf16.h>

#include "block_scale.cuh"
#include "common.cuh"
#include "tcgen05.cuh"

namespace epb {
namespace {

constexpr int BM = 128, BK = 128, UMMA_K = 32;      // BK in elements = bytes
constexpr int NT = 128;                             // most token rows of a tile: one scale chunk
constexpr int BOX_N = kNarrowFp8BoxRows;
constexpr int A_BYTES = 2 * BM * BK, STAGE_BYTES = A_BYTES + NT * BK;  // 48 KB
constexpr int SF_BYTES = 2048;                      // 512 B each: first block, second block, token rows
constexpr int STAGES = 4;
constexpr uint32_t TMEM_COLS = 512, kSfCol = 256;   // two accumulator blocks of NT columns, then two sets of 12 scale columns
constexpr int NUM_THREADS = 320;
constexpr int MAX_GROUPS = 320;
constexpr int kCtrlBytes = 1536;
constexpr int kStageHalfBytes = 32 * BM * 2;        // staging of four epilogue warps: 32 token rows x 128 features, bf16
constexpr int kAmaxBytes = 2 * 4 * 32 * 4;
constexpr size_t kSmemBytes = STAGES * (STAGE_BYTES + SF_BYTES) + 1024 + kCtrlBytes + 2 * kStageHalfBytes + kAmaxBytes;
static_assert(kSmemBytes <= 232448, "shared memory budget");
static_assert((STAGES * 2 + 2) * 8 + 8 + (MAX_GROUPS + 1) * 4 <= kCtrlBytes, "control block does not fit");

struct Tile {
  int mt, row, n, wslot;
};

// `g` is the caller's cursor; token tiles of one weight tile are neighbours.
__device__ __forceinline__ bool find_tile(const Fp8GemmArgs& a, int n_groups, const int* tile_prefix, int t, int& g, Tile& out) {
  while (g < n_groups && t >= tile_prefix[g + 1]) ++g;
  if (g >= n_groups) return false;
  const int rows = a.group_rows[g], nt_count = ceil_div(rows, NT);
  const int local = t - tile_prefix[g];
  out.mt = local / nt_count;
  const int nt = local - out.mt * nt_count;
  out.row = a.group_off[g] + nt * NT;
  out.n = min(NT, rows - nt * NT);
  out.wslot = a.group_wslot[g];
  return true;
}

template <bool kAct>
__global__ void __launch_bounds__(NUM_THREADS, 1)
narrow_gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                       const __grid_constant__ NarrowFp8Args args) {
  const Fp8GemmArgs& ga = args.g;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = smem;
  uint8_t* sf_tiles = smem + STAGES * STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sf_tiles + STAGES * SF_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* tile_prefix = abort_flag + 1;
  uint8_t* stage_tiles = sf_tiles + STAGES * SF_BYTES + kCtrlBytes;
  float* amax_tiles = reinterpret_cast<float*>(stage_tiles + 2 * kStageHalfBytes);  // [2 halves][4 warps][32 tokens]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_groups = min(ga.totals[1], ga.n_groups_cap);
  const int blocks = ga.N / BM;                       // 128-feature blocks of the output
  const int m_tiles = kAct ? blocks : ceil_div(blocks, 2);
  const int kblocks = ga.K / BK, kgroups = (kblocks + 3) / 4;
  const int w_blocks = kAct ? 2 * blocks : blocks;    // 128-row blocks of a weight slot

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 8);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  if (warp == 2) warp_tile_prefix(tile_prefix, n_groups, lane, [&](int g) { return ceil_div(ga.group_rows[g], NT) * m_tiles; });
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  volatile int* abort_v = abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0, cursor = 0;
      uint32_t phase = 0;
      Tile t, next;
      bool have = find_tile(ga, n_groups, tile_prefix, blockIdx.x, cursor, t), go = true;
      for (int ti = blockIdx.x; have && go && !*abort_v; ti += gridDim.x, t = next) {
        have = find_tile(ga, n_groups, tile_prefix, ti + gridDim.x, cursor, next);
        const int b0 = kAct ? t.mt : 2 * t.mt, b1 = kAct ? blocks + t.mt : b0 + 1;  // weight blocks of the tile
        const bool two = kAct || b1 < blocks;
        const int boxes = ceil_div(t.n, BOX_N);
        const uint8_t* sf0 = ga.sfb + ((size_t)t.wslot * w_blocks + b0) * kgroups * 512;
        const uint8_t* sf1 = ga.sfb + ((size_t)t.wslot * w_blocks + b1) * kgroups * 512;
        const uint8_t* sfx = ga.sfa + (size_t)(t.row / 128) * kgroups * 512;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_v, ga.status, 31)) {
            go = false;
            break;
          }
          uint8_t* sA = tiles + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          uint8_t* sS = sf_tiles + stage * SF_BYTES;
          uint64_t* fb = &full_bar[stage];
          const bool with_sf = (kb & 3) == 0;
          mbar_expect_tx(fb, (two ? A_BYTES : A_BYTES / 2) + boxes * BOX_N * BK + (with_sf ? (two ? 1536 : 1024) : 0));
          for (int r = 0; r < BM; r += args.w_box_rows) {
            tma_load_3d(sA + r * BK, &tmW, fb, kb * BK, b0 * BM + r, t.wslot);
            if (two) tma_load_3d(sA + (BM + r) * BK, &tmW, fb, kb * BK, b1 * BM + r, t.wslot);
          }
          for (int j = 0; j < boxes; ++j) tma_load_2d(sB + j * BOX_N * BK, &tmX, fb, kb * BK, t.row + j * BOX_N);
          if (with_sf) {
            bulk_load(sS, sf0 + (size_t)(kb >> 2) * 512, 512, fb);
            if (two) bulk_load(sS + 512, sf1 + (size_t)(kb >> 2) * 512, 512, fb);
            bulk_load(sS + 1024, sfx + (size_t)(kb >> 2) * 512, 512, fb);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ scale copies + MMA issue
    if (lane == 0) {
      int stage = 0, cursor = 0;
      uint32_t phase = 0, acc_phase = 0, sf_buf = 0;
      Tile t, next;
      bool have = find_tile(ga, n_groups, tile_prefix, blockIdx.x, cursor, t);
      for (int ti = blockIdx.x; have && !*abort_v; ti += gridDim.x, t = next) {
        have = find_tile(ga, n_groups, tile_prefix, ti + gridDim.x, cursor, next);
        const bool two = kAct || 2 * t.mt + 1 < blocks;
        const int ncols = round_up(t.n, 32);
        if (!mbar_wait(acc_empty, acc_phase ^ 1u, abort_v, ga.status, 32)) break;
        acc_phase ^= 1u;
        tc_fence_after();
        bool failed = false;
        uint32_t sf_w = 0;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_v, ga.status, 33)) {
            failed = true;
            break;
          }
          tc_fence_after();
          const uint32_t sA = smem_u32(tiles + stage * STAGE_BYTES), sB = sA + A_BYTES;
          if ((kb & 3) == 0) {
            // two sets of scale columns: the copies of one k-group never race the MMAs of the one before
            const uint32_t sS = smem_u32(sf_tiles + stage * SF_BYTES);
            sf_w = tmem_base + kSfCol + sf_buf * 16;
            tmem_cp_sf(sf_w, make_desc_sf(sS));
            if (two) tmem_cp_sf(sf_w + 4, make_desc_sf(sS + 512));
            tmem_cp_sf(sf_w + 8, make_desc_sf(sS + 1024));
            sf_buf ^= 1u;
          }
          const uint32_t id = (uint32_t)(kb & 3);
          const uint32_t idesc = make_idesc_scaled(ncols, BM, id, id);
          const uint64_t da = make_desc(sA, 16, 1024), db = make_desc(sB, 16, 1024);
          constexpr uint64_t a_block = (BM * BK) >> 4;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t step = (uint64_t)(k * (UMMA_K >> 4));
            const uint32_t acc = (kb | k) ? 1u : 0u;
            umma_fp8_scaled(tmem_base, da + step, db + step, idesc, sf_w, sf_w + 8, acc);
            if (two) umma_fp8_scaled(tmem_base + NT, da + a_block + step, db + step, idesc, sf_w + 4, sf_w + 8, acc);
          }
          umma_commit(&empty_bar[stage]);  // frees the stage (tiles and scale chunks) once read
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (failed) break;
        umma_commit(acc_full);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    // Lane = output feature, column = token; four warps (a half) cover 128 features.  kAct: the halves take 64 tokens each,
    // gate and up block; plain: each half takes one block, all tokens.
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    uint8_t* stg = stage_tiles + half * kStageHalfBytes;
    float* amax_half = amax_tiles + half * 128;
    uint32_t acc_phase = 0;
    int cursor = 0;
    Tile t;
    char* out0 = reinterpret_cast<char*>(ga.out);
    for (int ti = blockIdx.x; find_tile(ga, n_groups, tile_prefix, ti, cursor, t); ti += gridDim.x) {
      const bool ok = mbar_wait(acc_full, acc_phase, abort_v, ga.status, 34);
      if (!half_all(half, ok)) break;  // a half shares barriers: its warps leave together
      acc_phase ^= 1u;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
      const int chunks = ceil_div(t.n, 32);
      uint32_t v[4][32];
      if (kAct) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (half * 2 + i < chunks) {
            tmem_ld32(taddr + (half * 2 + i) * 32, v[i]);
            tmem_ld32(taddr + NT + (half * 2 + i) * 32, v[2 + i]);
          }
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (c < chunks) tmem_ld32(taddr + half * NT + c * 32, v[c]);
      }
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);  // the registers hold the tile: the next one may overwrite the buffer
      if (kAct) {
        const int kgroups_out = (blocks + 3) / 4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int c = half * 2 + i;
          if (c >= chunks) break;
          const int tok = c * 32 + lane;
          const size_t row = (size_t)t.row + tok;
          const bool real = tok < t.n && row < (size_t)ga.row_capacity;
          // activation from the bf16-rounded pre-activations, as the kernels with a pass of their own compute it
          float mine = 0.f;  // largest magnitude of token `lane` over this warp's features
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float g = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[i][j])));
            const float u = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[2 + i][j])));
            const float f = g * __fdividef(1.f, 1.f + __expf(-g)) * u;
            v[i][j] = __float_as_uint(f);
            // non-negative floats order like their bits; fmaxf drops a NaN
            const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(f), 0.f)));
            if (lane == j) mine = __uint_as_float(m);
          }
          half_sync(half);  // the previous chunk's flush has read the staging tile and the maxima
          amax_half[quarter * 32 + lane] = mine;
          half_sync(half);
          mine = fmaxf(fmaxf(amax_half[lane], amax_half[32 + lane]), fmaxf(amax_half[64 + lane], amax_half[96 + lane]));
          const int e = scale_exponent(mine);
          const float my_inv = exp2_int(-e);
#pragma unroll
          for (int j = 0; j < 32; ++j)
            stg[j * BM + quarter * 32 + lane] =
                __nv_cvt_float_to_fp8(__uint_as_float(v[i][j]) * __shfl_sync(0xffffffffu, my_inv, j), __NV_SATFINITE, __NV_E4M3);
          if (quarter == 0 && real)
            args.sf_out[(row >> 7) * kgroups_out * 512 + (size_t)(t.mt >> 2) * 512 + chunk_byte((int)(row & 127), t.mt)] = (uint8_t)(e + 127);
          half_sync(half);
          // 32 tokens x 128 B: a warp stores 8 tokens, four per instruction
          const unsigned long long p = real ? reinterpret_cast<unsigned long long>(args.q_out + row * (size_t)ga.N + t.mt * BM) : 0ull;
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int tk = quarter * 8 + it * 4 + (lane >> 3), piece = lane & 7;
            const unsigned long long base = __shfl_sync(0xffffffffu, p, tk);
            if (base != 0ull) *reinterpret_cast<uint4*>(base + piece * 16) = *reinterpret_cast<const uint4*>(stg + tk * BM + piece * 16);
          }
        }
      } else {
        const int block = 2 * t.mt + half;
        if (block < blocks) {  // the same for the whole half
          __nv_bfloat16* stg16 = reinterpret_cast<__nv_bfloat16*>(stg);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c >= chunks) break;
            const int tok = c * 32 + lane;
            const size_t row = (size_t)t.row + tok;
            char* orow = nullptr;
            if (tok < t.n && row < (size_t)ga.row_capacity) {
              if (ga.meta != nullptr) {
                const int2 mt = ga.meta[row];
                char* base = ga.out_ptrs ? reinterpret_cast<char*>(ga.out_ptrs[mt.x]) : out0;
                orow = base + (size_t)mt.y * ga.N * 2;
              } else {
                orow = out0 + row * (size_t)ga.N * 2;
              }
            }
            half_sync(half);
#pragma unroll
            for (int j = 0; j < 32; ++j) stg16[j * BM + quarter * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[c][j]));
            half_sync(half);
            const unsigned long long p = reinterpret_cast<unsigned long long>(orow);
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int tk = quarter * 8 + it * 2 + (lane >> 4), piece = lane & 15;
              const unsigned long long base = __shfl_sync(0xffffffffu, p, tk);
              if (base != 0ull) *reinterpret_cast<uint4*>(base + block * BM * 2 + piece * 16) = *reinterpret_cast<const uint4*>(stg + tk * BM * 2 + piece * 16);
            }
          }
        }
      }
    }
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_v && threadIdx.x == 0) {
    // let copies that were already issued land before the shared memory is released
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <bool kAct>
cudaError_t launch(const CUtensorMap& tmW, const CUtensorMap& tmX, const NarrowFp8Args& args, int num_sms, cudaStream_t stream) {
  static bool configured[kMaxTrackedDevices] = {};
  int dev;
  if (device_needs_setup(configured, &dev)) {
    cudaError_t e = cudaFuncSetAttribute(narrow_gemm_fp8_kernel<kAct>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return e;
    device_setup_done(configured, dev);
  }
  narrow_gemm_fp8_kernel<kAct><<<num_sms, NUM_THREADS, kSmemBytes, stream>>>(tmW, tmX, args);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_narrow_gemm_fp8(const CUtensorMap& tmW, const CUtensorMap& tmX, const NarrowFp8Args& args, int num_sms,
                                   cudaStream_t stream) {
  const Fp8GemmArgs& g = args.g;
  if (g.n_groups_cap > MAX_GROUPS || g.N % BM != 0 || g.K % BK != 0 || g.K <= 0) return cudaErrorInvalidValue;
  if ((args.w_box_rows != 64 && args.w_box_rows != 128) || (args.q_out == nullptr) != (args.sf_out == nullptr)) return cudaErrorInvalidValue;
  return args.q_out != nullptr ? launch<true>(tmW, tmX, args, num_sms, stream) : launch<false>(tmW, tmX, args, num_sms, stream);
}

}  // namespace epb
