// Block-scaled fp8 grouped GEMM: out[rows, N] = A_q[rows, K] * B_q[slot][N, K]^T with 1 x 128 activation
// scales and 128 x 128 weight scales applied by the tensor core (kind::mxf8f6f4.block_scale).
//
// One persistent CTA per SM, 320 threads:
//   warp 0      TMA producer: per k-block one 128 x 128-byte tile of A and of B (128-byte swizzle) and,
//               at every fourth k-block, the two 512-byte scale chunks (bulk copies on the same barrier)
//   warp 1      one thread copies the scale chunks shared -> tensor memory (tcgen05.cp) and issues four
//               128 x 128 x 32 MMAs per k-block; accumulators: two 128-column fp32 buffers in TMEM
//   warps 2-9   epilogue: tcgen05.ld, bf16 pack, staged 128-byte row stores (optionally to peer buffers)
// Every mbarrier wait is bounded; on a timeout the CTA raises its abort flag, records a status,
// lets issued copies land, frees its tensor memory and returns.
#include "grouped_gemm_fp8.h"

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "block_scale.cuh"
#include "common.cuh"
#include "tcgen05.cuh"

namespace epb {
namespace {

constexpr int BM = 128, BN = 128, BK = 128;       // BK in elements = bytes
constexpr int UMMA_K = 32;
constexpr int STAGES = 5;
constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK, TILE_BYTES = A_BYTES + B_BYTES;
constexpr int SF_BYTES = 1024;                     // 512 B for A + 512 B for B per stage
constexpr int NUM_THREADS = 320;
constexpr int MAX_GROUPS = 320;
constexpr int kCtrlBytes = 1536;
constexpr int kStageWarpBytes = 4096;
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t kSfCol = 256;                   // scale factors live behind the two accumulators
static_assert((STAGES * 2 + 4) * 8 + 8 + (MAX_GROUPS + 1) * 4 <= kCtrlBytes, "control block does not fit");

struct Tile {
  int g, mt, nt, rows, row0, wslot;
};

// `g` is the caller's cursor (0 before its first tile): tile indices only grow.  The producer and the MMA issuer look their
// next tile up before they work on the current one, as in grouped_gemm.cu.
__device__ __forceinline__ bool find_tile(const Fp8GemmArgs& a, int n_groups, int n_tiles_n, const int* tile_prefix,
                                          int t, int& g, Tile& out) {
  while (g < n_groups && t >= tile_prefix[g + 1]) ++g;
  if (g >= n_groups) return false;
  const int local = t - tile_prefix[g];
  out.g = g;
  out.mt = local / n_tiles_n;
  out.nt = local - out.mt * n_tiles_n;
  out.rows = a.group_rows[g];
  out.row0 = a.group_off[g];
  out.wslot = a.group_wslot[g];
  return true;
}

__device__ __forceinline__ void pack_row(const uint32_t (&r)[32], uint4 (&out)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[i].x = pack_bf16(__uint_as_float(r[8 * i + 0]), __uint_as_float(r[8 * i + 1]));
    out[i].y = pack_bf16(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
    out[i].z = pack_bf16(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
    out[i].w = pack_bf16(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
  }
}
// 32 rows x 128 B staging tile; piece p (16 B) of row r at r*8 + (p ^ (r & 7)): conflict-free for the
// row-wise writes and for the flush, which stores four rows x 128 contiguous bytes per instruction.
__device__ __forceinline__ int wide_index(int r, int p) { return r * 8 + (p ^ (r & 7)); }
__device__ __forceinline__ void wide_store_half(uint4* tile, int lane, const uint4 (&p)[4], int half) {
#pragma unroll
  for (int i = 0; i < 4; ++i) tile[wide_index(lane, half * 4 + i)] = p[i];
}
__device__ __forceinline__ void wide_flush(const uint4* tile, int lane, char* rowptr, int byte_off) {
  const unsigned long long mine = reinterpret_cast<unsigned long long>(rowptr);
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = it * 4 + (lane >> 3), p = lane & 7;
    const unsigned long long base = __shfl_sync(0xffffffffu, mine, r);
    if (base != 0ull) *reinterpret_cast<uint4*>(base + byte_off + p * 16) = tile[wide_index(r, p)];
  }
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                        Fp8GemmArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = smem;
  uint8_t* sf_tiles = smem + STAGES * TILE_BYTES;                       // [STAGES][1024]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sf_tiles + STAGES * SF_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* tile_prefix = abort_flag + 1;        // [MAX_GROUPS + 1]
  uint4* stage_tiles = reinterpret_cast<uint4*>(sf_tiles + STAGES * SF_BYTES + kCtrlBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int n_groups = args.totals[1];
  if (n_groups > args.n_groups_cap) n_groups = args.n_groups_cap;
  const int n_tiles_n = args.N / BN;
  const int kblocks = args.K / BK;
  const int kgroups = (kblocks + 3) / 4;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  if (warp == 2)
    warp_tile_prefix(tile_prefix, n_groups, lane, [&](int g) { return ceil_div(args.group_rows[g], BM) * n_tiles_n; });
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int total_tiles = tile_prefix[n_groups];
  volatile int* abort_v = abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    int stage = 0, cursor = 0;
    uint32_t phase = 0;
    Tile t, next;
    bool have = find_tile(args, n_groups, n_tiles_n, tile_prefix, blockIdx.x, cursor, t);
    for (int ti = blockIdx.x; have; ti += gridDim.x, t = next) {
      int go = 1;
      have = find_tile(args, n_groups, n_tiles_n, tile_prefix, ti + gridDim.x, cursor, next);
      if (lane == 0) {
        if (*abort_v) go = 0;
        if (go) {
          const int row_tile = (t.row0 + t.mt * BM) / BM;
          const uint8_t* sfa = args.sfa + (size_t)row_tile * kgroups * 512;
          const uint8_t* sfb = args.sfb + ((size_t)t.wslot * n_tiles_n + t.nt) * kgroups * 512;
          for (int kb = 0; kb < kblocks; ++kb) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_v, args.status, 11)) {
              go = 0;
              break;
            }
            uint8_t* sA = tiles + stage * TILE_BYTES;
            uint8_t* sB = sA + A_BYTES;
            uint64_t* fb = &full_bar[stage];
            const bool with_sf = (kb & 3) == 0;
            mbar_expect_tx(fb, TILE_BYTES + (with_sf ? SF_BYTES : 0));
            tma_load_2d(sA, &tmA, fb, kb * BK, t.row0 + t.mt * BM);
            tma_load_3d(sB, &tmB, fb, kb * BK, t.nt * BN, t.wslot);
            if (with_sf) {
              uint8_t* sS = sf_tiles + stage * SF_BYTES;
              bulk_load(sS, sfa + (size_t)(kb >> 2) * 512, 512, fb);
              bulk_load(sS + 512, sfb + (size_t)(kb >> 2) * 512, 512, fb);
            }
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      go = __shfl_sync(0xffffffffu, go, 0);
      if (!go) break;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ scale copies + MMA issue
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      int local = 0;
      uint32_t sf_buf = 0;  // two sets of scale columns: the copy for k-group g+1 never races the MMAs of g
      int cursor = 0;
      Tile t, next;
      bool have = find_tile(args, n_groups, n_tiles_n, tile_prefix, blockIdx.x, cursor, t);
      for (int ti = blockIdx.x; have && !*abort_v; ti += gridDim.x, ++local, t = next) {
        have = find_tile(args, n_groups, n_tiles_n, tile_prefix, ti + gridDim.x, cursor, next);
        const int buf = local & 1;
        if (!mbar_wait(&acc_empty[buf], acc_phase[buf] ^ 1u, abort_v, args.status, 12)) break;
        acc_phase[buf] ^= 1u;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
        bool failed = false;
        uint32_t sfa_col = 0, sfb_col = 0;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_v, args.status, 13)) {
            failed = true;
            break;
          }
          tc_fence_after();
          const uint32_t sA = smem_u32(tiles + stage * TILE_BYTES);
          const uint32_t sB = sA + A_BYTES;
          if ((kb & 3) == 0) {
            const uint32_t sS = smem_u32(sf_tiles + stage * SF_BYTES);
            sfa_col = tmem_base + kSfCol + sf_buf * 8;
            sfb_col = sfa_col + 4;
            tmem_cp_sf(sfa_col, make_desc_sf(sS));
            tmem_cp_sf(sfb_col, make_desc_sf(sS + 512));
            sf_buf ^= 1u;
          }
          const uint32_t id = (uint32_t)(kb & 3);
          const uint32_t idesc = make_idesc_scaled(BN, BM, id, id);
          const uint64_t da = make_desc(sA, 16, 1024), db = make_desc(sB, 16, 1024);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_fp8_scaled(tmem_d, da + (uint64_t)(k * (UMMA_K >> 4)), db + (uint64_t)(k * (UMMA_K >> 4)), idesc, sfa_col,
                            sfb_col, (kb | k) ? 1u : 0u);
          umma_commit(&empty_bar[stage]);  // frees the stage (tiles and scale chunks) once read
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (failed) break;
        umma_commit(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int quarter = warp & 3;      // TMEM lanes [32*quarter, +32)
    const int half = (warp - 2) >> 2;  // columns [64*half, +64) of the tile
    uint4* stg = stage_tiles + (warp - 2) * (kStageWarpBytes / 16);
    uint32_t acc_phase[2] = {0, 0};
    int local = 0, cursor = 0;
    Tile t;
    char* out0 = reinterpret_cast<char*>(args.out);
    for (int ti = blockIdx.x; ti < total_tiles && !*abort_v; ti += gridDim.x, ++local) {
      if (!find_tile(args, n_groups, n_tiles_n, tile_prefix, ti, cursor, t)) break;
      const int buf = local & 1;
      if (!mbar_wait(&acc_full[buf], acc_phase[buf], abort_v, args.status, 14)) break;
      acc_phase[buf] ^= 1u;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + half * 64);
      const int row_in_group = t.mt * BM + quarter * 32 + lane;
      const size_t row = (size_t)t.row0 + row_in_group;
      char* orow = nullptr;
      if (row_in_group < t.rows && row < (size_t)args.row_capacity) {
        if (args.meta != nullptr) {
          const int2 mt = args.meta[row];
          char* base = args.out_ptrs ? reinterpret_cast<char*>(args.out_ptrs[mt.x]) : out0;
          orow = base + (size_t)mt.y * args.N * 2;
        } else {
          orow = out0 + row * (size_t)args.N * 2;
        }
      }
      uint32_t v0[32], v1[32];
      tmem_ld32(taddr, v0);
      tmem_ld32(taddr + 32, v1);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);  // the values are in registers: the buffer is free
      uint4 p0[4], p1[4];
      pack_row(v0, p0);
      pack_row(v1, p1);
      __syncwarp();
      wide_store_half(stg, lane, p0, 0);
      wide_store_half(stg, lane, p1, 1);
      __syncwarp();
      wide_flush(stg, lane, orow, (t.nt * BN + half * 64) * 2);
    }
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_v && threadIdx.x == 0) {
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);  // issued copies land before smem is released
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ================================================================ CTA-pair variant (cta_group::2)
// A thread-block cluster of two SMs computes a 256 x 128 tile: each CTA stages its own 128 rows of A, its
// own 64 of the 128 weight rows (B) and the scale chunks it needs (its rows' SFA chunk and the whole SFB
// chunk), so per MMA a CTA reads 6 KB of shared memory instead of 8 KB and the tensor pipe is no longer fed at
// the shared-memory limit.  Every load is a plain TMA load (no multicast) that completes on the barrier of
// the pair's even CTA; that CTA issues the scale copies and the MMAs for both.
namespace pair {

constexpr int kPairStageBytes = 2048;  // staging tile of one epilogue warp: 16 rows x 128 B, or 32 rows x 64 B

// 128 bytes of each lane's row (p0, then p1) to memory, 16 rows at a time, four rows x 128 contiguous bytes per instruction.
__device__ __forceinline__ void rows_out(uint4* tile, int lane, const uint4 (&p0)[4], const uint4 (&p1)[4], char* rowptr, int byte_off) {
  const unsigned long long mine = reinterpret_cast<unsigned long long>(rowptr);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    __syncwarp();
    if ((lane >> 4) == h) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        tile[wide_index(lane & 15, i)] = p0[i];
        tile[wide_index(lane & 15, 4 + i)] = p1[i];
      }
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int r = it * 4 + (lane >> 3), p = lane & 7;
      const unsigned long long base = __shfl_sync(0xffffffffu, mine, h * 16 + r);
      if (base != 0ull) *reinterpret_cast<uint4*>(base + byte_off + p * 16) = tile[wide_index(r, p)];
    }
  }
}

// kBN = 128: two accumulator buffers (epilogue overlaps the next tile).  kBN = 256: one 256-column accumulator
// (the scale factors need the rest of tensor memory), twice the MMA work per TMA load and per barrier round.
template <int kBN>
struct Geo {
  static constexpr int B_HALF = kBN / 2;                     // weight rows staged per CTA
  static constexpr int A_BYTES = BM * BK, B_BYTES = B_HALF * BK, TILE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SF_BYTES = 512 + 512 * (kBN / 128);   // this CTA's SFA chunk + the SFB chunks of the whole tile
  // A stage holds kSub k-blocks: a tcgen05.commit costs the tensor pipe idle cycles (ragged_gemm.cu), so there is one per stage.
  static constexpr int kSub = 2;
  static constexpr int STAGES = 3;
  static constexpr int STAGE_BYTES = kSub * TILE_BYTES;
  static constexpr int ACC_BUFS = kBN == 128 ? 2 : 1;
  static constexpr size_t SMEM = STAGES * (STAGE_BYTES + 2048) + 1024 + kCtrlBytes + 8 * kPairStageBytes + 1024 /*row maxima*/;
};
constexpr int TILE_M = 2 * BM;

__device__ __forceinline__ void tmem_cp_sf2(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma2(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t sfa,
                                      uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}

// Meeting point of the two epilogue warps that share 32 rows.
__device__ __forceinline__ void rows_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); }

// The same, and true if `ok` holds in both.
__device__ __forceinline__ bool rows_all(int quarter, bool ok) {
  uint32_t all;
  asm volatile(
      "{\n.reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "bar.red.and.pred q, %2, 64, p;\n"
      "selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(all)
      : "r"(ok ? 1u : 0u), "r"(1 + quarter)
      : "memory");
  return all != 0u;
}

// kAct (kBN = 256): a tile is 128 gate columns and their 128 up columns -- exactly one scale block of every row's activation --
// so SwiGLU and the quantisation happen here and the pre-activations (2 F bf16 values a row, written and read back) never
// reach memory.  Each CTA of the pair stages one of the two halves.  4096 tokens, 32 experts of 7168 x 2048: the layer
// 2301 -> 2249 us, without the pass of its own (75 us) and its 400 MB.
template <int kBN, bool kAct>
__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                             const __grid_constant__ CUtensorMap tmSFA, const __grid_constant__ CUtensorMap tmSFB,
                             Fp8GemmArgs args) {
  using G = Geo<kBN>;
  constexpr int STAGES = G::STAGES, TILE_BYTES = G::TILE_BYTES, A_BYTES = G::A_BYTES, B_HALF = G::B_HALF;
  constexpr int kSub = G::kSub, STAGE_BYTES = G::STAGE_BYTES;
  constexpr int SF_BYTES = 2048;   // slot size; G::SF_BYTES of it are used
  constexpr int ACC_BUFS = G::ACC_BUFS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = smem;
  uint8_t* sf_tiles = smem + STAGES * STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sf_tiles + STAGES * SF_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* tile_prefix = abort_flag + 1;
  uint4* stage_tiles = reinterpret_cast<uint4*>(sf_tiles + STAGES * SF_BYTES + kCtrlBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cta_rank = (int)cluster_ctarank();
  const int tile_first = blockIdx.x / 2, tile_stride = gridDim.x / 2;
  int n_groups = args.totals[1];
  if (n_groups > args.n_groups_cap) n_groups = args.n_groups_cap;
  const int n_tiles_n = args.N / (kAct ? 128 : kBN);
  const int n128 = args.N / 128 * (kAct ? 2 : 1);  // 128-row blocks of a weight slot
  const int kblocks = args.K / BK;
  const int kgroups = (kblocks + 3) / 4;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 16);   // 8 epilogue warps of each CTA
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, TMEM_COLS);
  if (warp == 2)
    warp_tile_prefix(tile_prefix, n_groups, lane, [&](int g) { return ceil_div(args.group_rows[g], TILE_M) * n_tiles_n; });
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int total_tiles = tile_prefix[n_groups];
  volatile int* abort_v = abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs)
    int stage = 0, cursor = 0;
    uint32_t phase = 0;
    Tile t, next;
    bool have = find_tile(args, n_groups, n_tiles_n, tile_prefix, tile_first, cursor, t);
    for (int ti = tile_first; have; ti += tile_stride, t = next) {
      int go = 1;
      have = find_tile(args, n_groups, n_tiles_n, tile_prefix, ti + tile_stride, cursor, next);
      if (lane == 0) {
        if (*abort_v) go = 0;
        if (go) {
          const int row_first = t.row0 + t.mt * TILE_M + cta_rank * BM;
          const int sfa_chunk = (row_first / BM) * kgroups;
          const int sfb_chunk = (t.wslot * n128 + t.nt * (kAct ? 1 : kBN / 128)) * kgroups;
          const int sfb_step = (kAct ? args.N / 128 : 1) * kgroups;  // from the tile's first scale block to its second
          const int b_row = kAct ? cta_rank * args.N + t.nt * 128 : t.nt * kBN + cta_rank * B_HALF;
          for (int kb0 = 0; kb0 < kblocks; kb0 += kSub) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_v, args.status, 21)) {
              go = 0;
              break;
            }
            uint64_t* fb = &full_bar[stage];
            const int subs = min(kSub, kblocks - kb0);
            const bool with_sf = (kb0 & 3) == 0;
            if (cta_rank == 0) mbar_expect_tx(fb, 2 * (subs * TILE_BYTES + (with_sf ? G::SF_BYTES : 0)));
            for (int sub = 0; sub < subs; ++sub) {
              uint8_t* sA = tiles + stage * STAGE_BYTES + sub * TILE_BYTES;
              tma_load_2d_pair(sA, &tmA, fb, (kb0 + sub) * BK, row_first);
              tma_load_3d_pair(sA + A_BYTES, &tmB, fb, (kb0 + sub) * BK, b_row, t.wslot);
            }
            if (with_sf) {
              uint8_t* sS = sf_tiles + stage * SF_BYTES;
              tma_load_2d_pair(sS, &tmSFA, fb, 0, sfa_chunk + (kb0 >> 2));
#pragma unroll
              for (int j = 0; j < kBN / 128; ++j)
                tma_load_2d_pair(sS + 512 + 512 * j, &tmSFB, fb, 0, sfb_chunk + j * sfb_step + (kb0 >> 2));
            }
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      go = __shfl_sync(0xffffffffu, go, 0);
      if (!go) break;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ scale copies + MMA issue (even CTA only)
    if (lane == 0 && cta_rank == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      int local = 0;
      uint32_t sf_buf = 0;
      int cursor = 0;
      Tile t, next;
      bool have = find_tile(args, n_groups, n_tiles_n, tile_prefix, tile_first, cursor, t);
      for (int ti = tile_first; have && !*abort_v; ti += tile_stride, ++local, t = next) {
        have = find_tile(args, n_groups, n_tiles_n, tile_prefix, ti + tile_stride, cursor, next);
        const int buf = ACC_BUFS == 2 ? (local & 1) : 0;
        if (!mbar_wait(&acc_empty[buf], acc_phase[buf] ^ 1u, abort_v, args.status, 22)) break;
        acc_phase[buf] ^= 1u;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * 128);
        bool failed = false;
        uint32_t sfa_col = 0, sfb_col = 0;
        for (int kb0 = 0; kb0 < kblocks; kb0 += kSub) {
          if (!mbar_wait(&full_bar[stage], phase, abort_v, args.status, 23)) {
            failed = true;
            break;
          }
          tc_fence_after();
          if ((kb0 & 3) == 0) {
            const uint32_t sS = smem_u32(sf_tiles + stage * SF_BYTES);
            sfa_col = tmem_base + kSfCol + sf_buf * 16;
            sfb_col = sfa_col + 4;
            tmem_cp_sf2(sfa_col, make_desc_sf(sS));
#pragma unroll
            for (int j = 0; j < kBN / 128; ++j) tmem_cp_sf2(sfb_col + 4 * j, make_desc_sf(sS + 512 + 512 * j));
            sf_buf ^= 1u;
          }
          const int subs = min(kSub, kblocks - kb0);
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub) {
            if (sub >= subs) break;
            const uint32_t sA = smem_u32(tiles + stage * STAGE_BYTES + sub * TILE_BYTES);
            const uint32_t id = (uint32_t)((kb0 + sub) & 3);
            const uint32_t idesc = make_idesc_scaled(kBN, TILE_M, id, id);
            const uint64_t da = make_desc(sA, 16, 1024), db = make_desc(sA + A_BYTES, 16, 1024);
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma2(tmem_d, da + (uint64_t)(k * (UMMA_K >> 4)), db + (uint64_t)(k * (UMMA_K >> 4)), idesc, sfa_col, sfb_col,
                    (kb0 | sub | k) ? 1u : 0u);
          }
          umma_commit_both(&empty_bar[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (failed) break;
        umma_commit_both(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9 of both CTAs)
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    uint4* stg = stage_tiles + (warp - 2) * (kPairStageBytes / 16);
    uint32_t acc_phase[2] = {0, 0};
    int local = 0, cursor = 0;
    Tile t;
    char* out0 = reinterpret_cast<char*>(args.out);
    for (int ti = tile_first; ti < total_tiles && (kAct || !*abort_v); ti += tile_stride, ++local) {
      if (!find_tile(args, n_groups, n_tiles_n, tile_prefix, ti, cursor, t)) break;
      const int buf = ACC_BUFS == 2 ? (local & 1) : 0;
      bool ok = mbar_wait(&acc_full[buf], acc_phase[buf], abort_v, args.status, 24);
      if (kAct) ok = rows_all(quarter, ok);  // two warps that share barriers leave together
      if (!ok) break;
      acc_phase[buf] ^= 1u;
      tc_fence_after();
      constexpr int COLS_PER_WARP = kBN / 2;                      // 64 or 128 columns per warp
      // kAct: 64 gate columns and their 64 up columns
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 128 + half * (kAct ? 64 : COLS_PER_WARP));
      const int row_in_group = t.mt * TILE_M + cta_rank * BM + quarter * 32 + lane;
      const size_t row = (size_t)t.row0 + row_in_group;
      char* orow = nullptr;
      if (!kAct && row_in_group < t.rows && row < (size_t)args.row_capacity) {
        if (args.meta != nullptr) {
          const int2 mt = args.meta[row];
          char* base = args.out_ptrs ? reinterpret_cast<char*>(args.out_ptrs[mt.x]) : out0;
          orow = base + (size_t)mt.y * args.N * 2;
        } else {
          orow = out0 + row * (size_t)args.N * 2;
        }
      }
      // read this warp's whole share of the accumulator into registers first and hand the buffer back at once:
      // with a single accumulator the next tile's MMAs wait for exactly this read
      uint32_t v[COLS_PER_WARP / 32][32];
#pragma unroll
      for (int c = 0; c < COLS_PER_WARP / 32; ++c) tmem_ld32(taddr + (kAct ? (c & 1) * 32 + (c >> 1) * 128 : c * 32), v[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[buf]), 0));
      if (kAct) {
        const bool real = row_in_group < t.rows && row < (size_t)args.row_capacity;
        float amax = 0.f;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            // activation from the bf16-rounded pre-activations, as the pass of its own computes it
            const float g = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[c][j])));
            const float u = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[COLS_PER_WARP / 32 - 2 + c][j])));
            const float f = g * __fdividef(1.f, 1.f + __expf(-g)) * u;
            v[c][j] = __float_as_uint(f);
            amax = fmaxf(amax, fabsf(f));
          }
        }
        // the row's other 64 features are in the warp that shares its quarter
        float* maxima = reinterpret_cast<float*>(stage_tiles + 8 * (kPairStageBytes / 16)) + quarter * 64;
        maxima[half * 32 + lane] = amax;
        rows_sync(quarter);
        amax = fmaxf(amax, maxima[(half ^ 1) * 32 + lane]);
        const int e = scale_exponent(amax);
        const float inv = exp2_int(-e);
        if (half == 0 && real)
          args.sf_out[(row >> 7) * (size_t)((args.N / 128 + 3) / 4) * 512 + (size_t)(t.nt >> 2) * 512 + chunk_byte((int)(row & 127), t.nt)] =
              (uint8_t)(e + 127);
        uint4 q[4];
        uint32_t* qw = reinterpret_cast<uint32_t*>(q);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t* w = &v[i >> 3][(i & 7) * 4];
          const unsigned lo = __nv_cvt_float2_to_fp8x2(make_float2(__uint_as_float(w[0]) * inv, __uint_as_float(w[1]) * inv), __NV_SATFINITE, __NV_E4M3);
          const unsigned hi = __nv_cvt_float2_to_fp8x2(make_float2(__uint_as_float(w[2]) * inv, __uint_as_float(w[3]) * inv), __NV_SATFINITE, __NV_E4M3);
          qw[i] = (lo & 0xffffu) | (hi << 16);
        }
        // 32 rows x 64 B through the staging tile (piece p of row r at r * 4 + (p ^ ((r >> 1) & 3)): no bank conflicts), then
        // 8 rows x 64 contiguous bytes per instruction
        __syncwarp();
#pragma unroll
        for (int p = 0; p < 4; ++p) stg[lane * 4 + (p ^ ((lane >> 1) & 3))] = q[p];
        __syncwarp();
        const unsigned long long mine =
            real ? reinterpret_cast<unsigned long long>(args.q_out + row * (size_t)args.N + t.nt * 128 + half * 64) : 0ull;
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int r = it * 8 + (lane >> 2), p = lane & 3;
          const unsigned long long base = __shfl_sync(0xffffffffu, mine, r);
          if (base != 0ull) *reinterpret_cast<uint4*>(base + p * 16) = stg[r * 4 + (p ^ ((r >> 1) & 3))];
        }
        rows_sync(quarter);  // the maxima may be overwritten
      } else {
#pragma unroll
        for (int pairc = 0; pairc < COLS_PER_WARP / 64; ++pairc) {
          uint4 p0[4], p1[4];
          pack_row(v[2 * pairc], p0);
          pack_row(v[2 * pairc + 1], p1);
          rows_out(stg, lane, p0, p1, orow, (t.nt * kBN + half * COLS_PER_WARP + pairc * 64) * 2);
        }
      }
    }
  }

  __syncthreads();
  if (*abort_v && threadIdx.x == 0) {
    unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

static_assert(Geo<128>::SMEM <= 232448 && Geo<256>::SMEM <= 232448, "shared memory budget exceeded");

}  // namespace pair

constexpr size_t kSmemBytes = STAGES * TILE_BYTES + STAGES * SF_BYTES + 1024 + kCtrlBytes + 8 * kStageWarpBytes;
static_assert(kSmemBytes <= 232448, "shared memory budget exceeded");

// ---------------------------------------------------------------- quantisers
// Is `row` inside one of the groups?  The whole warp calls this with the same row.
__device__ __forceinline__ bool row_is_real(const RowGroups& g, int row, int lane) {
  if (g.group_off == nullptr) return true;
  if (row >= g.totals[0]) return false;
  int n = g.totals[1];
  if (n > g.n_groups_cap) n = g.n_groups_cap;
  for (int base = 0; base < n; base += 32) {
    const int i = base + lane;
    const bool in = i < n && row >= g.group_off[i] && row < g.group_off[i] + g.group_rows[i];
    if (__ballot_sync(0xffffffffu, in)) return true;
  }
  return false;
}

// One warp per row; per 128-wide block each lane handles 4 consecutive values.
__global__ void __launch_bounds__(256) quantize_rows_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                                                            uint8_t* __restrict__ sfa, int rows, int K, RowGroups groups) {
  const int warp = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (warp >= rows || !row_is_real(groups, warp, lane)) return;
  const int kblocks = K / 128, kgroups = (kblocks + 3) / 4;
  const __nv_bfloat16* xr = x + (size_t)warp * K;
  uint8_t* qr = q + (size_t)warp * K;
  uint8_t* chunk_row = sfa + (size_t)(warp >> 7) * kgroups * 512;
  for (int kb = 0; kb < kblocks; ++kb) {
    const uint2 raw = *reinterpret_cast<const uint2*>(xr + kb * 128 + lane * 4);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    float amax = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const int e = scale_exponent(amax);
    const float inv = exp2_int(-e);
    const unsigned lo = __nv_cvt_float2_to_fp8x2(make_float2(a.x * inv, a.y * inv), __NV_SATFINITE, __NV_E4M3);
    const unsigned hi = __nv_cvt_float2_to_fp8x2(make_float2(b.x * inv, b.y * inv), __NV_SATFINITE, __NV_E4M3);
    *reinterpret_cast<uint32_t*>(qr + kb * 128 + lane * 4) = (lo & 0xffffu) | (hi << 16);
    if (lane == 0) chunk_row[(size_t)(kb >> 2) * 512 + chunk_byte(warp & 127, kb)] = (uint8_t)(e + 127);
  }
  // k-blocks of a partial last group keep the neutral exponent
  if (lane == 0)
    for (int kb = kblocks; kb < kgroups * 4; ++kb) chunk_row[(size_t)(kb >> 2) * 512 + chunk_byte(warp & 127, kb)] = 127;
}

// One warp per token and 1024-wide piece of its row: the piece is read and quantised ONCE and stored to all topk destinations
// (peer memory).  A 128-wide block is held by 16 lanes (8 values each); the block maximum is a 4-step shuffle inside the
// half-warp.  The four loads of a piece are issued together.  Bound by the topk stores: 4096 tokens x 8 x 7168 in 113 us
// (2.1 TB/s) with one warp per routed unit, which read and quantised every token eight times, 50 now; 64 tokens 12.7 -> 5.2.
constexpr int kDispatchVecs = 4;  // 16-byte vectors of a row that a lane holds
__global__ void __launch_bounds__(256) dispatch_fp8_kernel(DispatchFp8Args a, int num_tokens, int pieces) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const long long item = (long long)blockIdx.x * wpb + warp;
  const int t = (int)(item / pieces), piece = (int)(item - (long long)t * pieces);
  if (t >= num_tokens) return;
  const int vec_per_row = a.H / 8;
  const int kgroups = (a.H / 128 + 3) / 4;
  const uint4* src = reinterpret_cast<const uint4*>(a.rows) + (size_t)t * vec_per_row;
  uint4 raw[kDispatchVecs];
#pragma unroll
  for (int i = 0; i < kDispatchVecs; ++i) {
    const int v = (piece * kDispatchVecs + i) * 32 + lane;
    raw[i] = v < vec_per_row ? src[v] : make_uint4(0, 0, 0, 0);
  }
  uint2 q[kDispatchVecs];
  uint8_t exps[kDispatchVecs];
#pragma unroll
  for (int i = 0; i < kDispatchVecs; ++i) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[i]);
    float f[8];
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 p = __bfloat1622float2(h[j]);
      f[2 * j] = p.x;
      f[2 * j + 1] = p.y;
      amax = fmaxf(amax, fmaxf(fabsf(p.x), fabsf(p.y)));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const int e = scale_exponent(amax);
    const float inv = exp2_int(-e);
    uint32_t out[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j] * inv, f[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      const unsigned hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j + 2] * inv, f[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
      out[j] = (lo & 0xffffu) | (hi << 16);
    }
    q[i] = make_uint2(out[0], out[1]);
    exps[i] = (uint8_t)(e + 127);
  }
  for (int k0 = 0; k0 < a.topk; k0 += 32) {
    // lane k holds the destination of the token's unit k0 + k
    int my_dst = -1, my_row = 0;
    if (k0 + lane < a.topk) {
      const int u = t * a.topk + k0 + lane;
      my_dst = a.unit_dst[u];
      my_row = a.unit_row[u];
      if (my_row >= a.row_capacity) my_dst = -1;
      if (piece == 0 && my_dst >= 0 && a.meta_ptrs != nullptr) a.meta_ptrs[my_dst][my_row] = make_int2(a.me, a.unit_pos[u]);
    }
    const int n = min(32, a.topk - k0);
    for (int k = 0; k < n; ++k) {
      const int dst = __shfl_sync(0xffffffffu, my_dst, k), row = __shfl_sync(0xffffffffu, my_row, k);
      if (dst < 0) continue;
      uint8_t* qrow = a.xq_ptrs[dst] + (size_t)row * a.H;
      uint8_t* chunk_row = a.sfx_ptrs[dst] + (size_t)(row >> 7) * kgroups * 512;
#pragma unroll
      for (int i = 0; i < kDispatchVecs; ++i) {
        const int v = (piece * kDispatchVecs + i) * 32 + lane;
        if (v >= vec_per_row) continue;
        *reinterpret_cast<uint2*>(qrow + (size_t)v * 8) = q[i];
        const int kb = v >> 4;
        if ((lane & 15) == 0) chunk_row[(size_t)(kb >> 2) * 512 + chunk_byte(row & 127, kb)] = exps[i];
      }
    }
  }
}

// SwiGLU + quantisation in one pass: h [rows, 2F] (gate columns, then up columns) ->
// act = silu(gate) * up as e4m3 [rows, F] with 1 x 128 scales (and, optionally, as bf16 too).
__global__ void __launch_bounds__(256) swiglu_quantize_kernel(const __nv_bfloat16* __restrict__ h, uint8_t* __restrict__ q,
                                                              uint8_t* __restrict__ sfa, __nv_bfloat16* __restrict__ act,
                                                              int rows, int F, RowGroups groups) {
  const int warp = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (warp >= rows || !row_is_real(groups, warp, lane)) return;
  // A half-warp holds a 128-wide block (8 values per lane), a pass of the loop kUnroll x 256 columns: all its loads are
  // issued before the first is used (512 rows of 2048: 16 us with 8-byte loads and one block per pass, 8.8 now; 32768 rows
  // 85 -> 75).
  const int kblocks = F / 128, kgroups = (kblocks + 3) / 4, vec_per_row = F / 8;
  const uint4* gr = reinterpret_cast<const uint4*>(h + (size_t)warp * 2 * F);
  const uint4* ur = gr + vec_per_row;
  uint8_t* qr = q + (size_t)warp * F;
  uint8_t* chunk_row = sfa + (size_t)(warp >> 7) * kgroups * 512;
  constexpr int kUnroll = 4;
  for (int v0 = 0; v0 < vec_per_row; v0 += 32 * kUnroll) {
    uint4 graw[kUnroll], uraw[kUnroll];
#pragma unroll
    for (int i = 0; i < kUnroll; ++i) {
      const int v = v0 + i * 32 + lane;
      graw[i] = v < vec_per_row ? gr[v] : make_uint4(0, 0, 0, 0);
      uraw[i] = v < vec_per_row ? ur[v] : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < kUnroll; ++i) {
      const int v = v0 + i * 32 + lane;
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&graw[i]);
      const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&uraw[i]);
      float f[8];
      float amax = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 g = __bfloat1622float2(gh[j]), u = __bfloat1622float2(uh[j]);
        f[2 * j] = g.x * __fdividef(1.f, 1.f + __expf(-g.x)) * u.x;
        f[2 * j + 1] = g.y * __fdividef(1.f, 1.f + __expf(-g.y)) * u.y;
        amax = fmaxf(amax, fmaxf(fabsf(f[2 * j]), fabsf(f[2 * j + 1])));
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      if (v >= vec_per_row) continue;
      if (act != nullptr)
        *reinterpret_cast<uint4*>(act + (size_t)warp * F + (size_t)v * 8) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
      const int e = scale_exponent(amax);
      const float inv = exp2_int(-e);
      uint32_t out[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const unsigned lo = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j] * inv, f[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
        const unsigned hi = __nv_cvt_float2_to_fp8x2(make_float2(f[4 * j + 2] * inv, f[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
        out[j] = (lo & 0xffffu) | (hi << 16);
      }
      *reinterpret_cast<uint2*>(qr + (size_t)v * 8) = make_uint2(out[0], out[1]);
      const int kb = v >> 4;
      if ((lane & 15) == 0) chunk_row[(size_t)(kb >> 2) * 512 + chunk_byte(warp & 127, kb)] = (uint8_t)(e + 127);
    }
  }
}

// One CTA per (k-block, n-block, slot): 128 x 128 values, 256 threads, 64 values each.
__global__ void __launch_bounds__(256) quantize_weights_kernel(const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q,
                                                               uint8_t* __restrict__ sfb, int N, int K) {
  const int kb = blockIdx.x, nb = blockIdx.y, slot = blockIdx.z;
  const int kblocks = K / 128, kgroups = (kblocks + 3) / 4, n_tiles = N / 128;
  const size_t base = ((size_t)slot * N + (size_t)nb * 128) * K + (size_t)kb * 128;
  // thread t: row t/2 of the block, 64 consecutive values starting at (t%2)*64
  const int r = threadIdx.x >> 1, c0 = (threadIdx.x & 1) * 64;
  const uint4* src = reinterpret_cast<const uint4*>(w + base + (size_t)r * K + c0);
  uint4 v[8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = src[i];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
  }
  __shared__ float red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
  const int e = scale_exponent(amax);
  const float inv = exp2_int(-e);
  uint8_t* dst = q + base + (size_t)r * K + c0;
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    uint32_t out[4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[i + half]);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const float2 f0 = __bfloat1622float2(h[j]), f1 = __bfloat1622float2(h[j + 1]);
        const unsigned lo = __nv_cvt_float2_to_fp8x2(make_float2(f0.x * inv, f0.y * inv), __NV_SATFINITE, __NV_E4M3);
        const unsigned hi = __nv_cvt_float2_to_fp8x2(make_float2(f1.x * inv, f1.y * inv), __NV_SATFINITE, __NV_E4M3);
        out[half * 2 + j / 2] = (lo & 0xffffu) | (hi << 16);
      }
    }
    *reinterpret_cast<uint4*>(dst + i * 8) = make_uint4(out[0], out[1], out[2], out[3]);
  }
  uint8_t* chunk = sfb + (((size_t)slot * n_tiles + nb) * kgroups + (kb >> 2)) * 512;
  if (threadIdx.x < 128) chunk[chunk_byte(threadIdx.x, kb)] = (uint8_t)(e + 127);
  if (kb == kblocks - 1 && threadIdx.x < 128)
    for (int k2 = kblocks; k2 < kgroups * 4; ++k2) chunk[chunk_byte(threadIdx.x, k2)] = 127;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

}  // namespace

bool make_tmap_fp8_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_tmap_fp8_3d(CUtensorMap* out, const void* base, uint64_t slots, uint64_t rows, uint64_t cols,
                      uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[3] = {cols, rows, slots};
  cuuint64_t strides[2] = {cols, rows * cols};
  cuuint32_t box[3] = {128, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_tmap_sf(CUtensorMap* out, const void* base, uint64_t chunks) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr || chunks == 0) return false;
  cuuint64_t dims[2] = {128, chunks};          // one 512-byte chunk = 128 x int32
  cuuint64_t strides[1] = {512};
  cuuint32_t box[2] = {128, 1};
  cuuint32_t estr[2] = {1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_grouped_gemm_fp8_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmSFA,
                                         const CUtensorMap& tmSFB, const Fp8GemmArgs& args, int num_sms,
                                         cudaStream_t stream) {
  if (args.n_groups_cap > MAX_GROUPS || args.N % BN != 0 || args.K % BK != 0 || args.K <= 0) return cudaErrorInvalidValue;
  if ((args.q_out == nullptr) != (args.sf_out == nullptr)) return cudaErrorInvalidValue;
  const bool act = args.q_out != nullptr;
  const bool wide = act || args.N % 256 == 0;   // 256-column tiles when the width allows it
  static bool configured[kMaxTrackedDevices] = {};
  int dev;
  if (device_needs_setup(configured, &dev)) {
    cudaError_t e = cudaFuncSetAttribute(pair::grouped_gemm_fp8_pair_kernel<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)pair::Geo<128>::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(pair::grouped_gemm_fp8_pair_kernel<256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)pair::Geo<256>::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(pair::grouped_gemm_fp8_pair_kernel<256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)pair::Geo<256>::SMEM);
    if (e != cudaSuccess) return e;
    device_setup_done(configured, dev);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(num_sms / 2 * 2));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = wide ? pair::Geo<256>::SMEM : pair::Geo<128>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (act) return cudaLaunchKernelEx(&cfg, pair::grouped_gemm_fp8_pair_kernel<256, true>, tmA, tmB, tmSFA, tmSFB, args);
  if (wide) return cudaLaunchKernelEx(&cfg, pair::grouped_gemm_fp8_pair_kernel<256, false>, tmA, tmB, tmSFA, tmSFB, args);
  return cudaLaunchKernelEx(&cfg, pair::grouped_gemm_fp8_pair_kernel<128, false>, tmA, tmB, tmSFA, tmSFB, args);
}

cudaError_t launch_grouped_gemm_fp8(const CUtensorMap& tmA, const CUtensorMap& tmB, const Fp8GemmArgs& args,
                                    int num_sms, cudaStream_t stream) {
  if (args.n_groups_cap > MAX_GROUPS || args.N % BN != 0 || args.K % BK != 0 || args.K <= 0) return cudaErrorInvalidValue;
  static bool configured[kMaxTrackedDevices] = {};
  int dev;
  if (device_needs_setup(configured, &dev)) {
    cudaError_t e = cudaFuncSetAttribute(grouped_gemm_fp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSmemBytes);
    if (e != cudaSuccess) return e;
    device_setup_done(configured, dev);
  }
  grouped_gemm_fp8_kernel<<<num_sms, NUM_THREADS, kSmemBytes, stream>>>(tmA, tmB, args);
  return cudaGetLastError();
}

cudaError_t launch_quantize_rows(const void* x, uint8_t* q, uint8_t* sfa, int rows, int K, const RowGroups* groups,
                                 cudaStream_t stream) {
  if (rows % 128 != 0 || K % 128 != 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  const int blocks = (rows + 7) / 8;
  quantize_rows_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(x), q, sfa, rows, K,
                                                   groups ? *groups : RowGroups{nullptr, nullptr, nullptr, 0});
  return cudaGetLastError();
}

cudaError_t launch_dispatch_fp8(const DispatchFp8Args& a, cudaStream_t stream) {
  if (a.H % 128 != 0) return cudaErrorInvalidValue;
  if (a.num_units <= 0) return cudaSuccess;
  if (a.topk < 1 || a.num_units % a.topk != 0) return cudaErrorInvalidValue;
  const int wpb = 8, tokens = a.num_units / a.topk, pieces = ceil_div(a.H, kDispatchVecs * 256);
  const long long items = (long long)tokens * pieces;
  dispatch_fp8_kernel<<<(unsigned)((items + wpb - 1) / wpb), wpb * 32, 0, stream>>>(a, tokens, pieces);
  return cudaGetLastError();
}

cudaError_t launch_swiglu_quantize(const void* h, uint8_t* q, uint8_t* sfa, void* act, int rows, int F,
                                   const RowGroups* groups, cudaStream_t stream) {
  if (rows % 128 != 0 || F % 128 != 0) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  const int blocks = (rows + 7) / 8;
  swiglu_quantize_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(h), q, sfa,
                                                     reinterpret_cast<__nv_bfloat16*>(act), rows, F,
                                                     groups ? *groups : RowGroups{nullptr, nullptr, nullptr, 0});
  return cudaGetLastError();
}

cudaError_t launch_quantize_weights(const void* w, uint8_t* q, uint8_t* sfb, int slots, int N, int K,
                                    cudaStream_t stream) {
  if (N % 128 != 0 || K % 128 != 0) return cudaErrorInvalidValue;
  dim3 grid(K / 128, N / 128, slots);
  quantize_weights_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(w), q, sfb, N, K);
  return cudaGetLastError();
}

}  // namespace epb
