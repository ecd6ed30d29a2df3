// Grouped GEMM for few rows per expert: the WEIGHTS are the 128-row operand of the tensor core, the token rows are
// its N columns.
//
// Launches of 4 or 100 rows an expert are bound by reading the weights once from HBM.  Here one CTA's tile is 256 weight rows
// (output features) x up to 128 token rows, N is the real row count rounded up to 16, and every byte that the ring keeps in
// flight beyond a few KB is a weight byte (the CTA-pair kernel of ragged_gemm.cu brings a box of 128 token rows a CTA whatever
// the tile holds).  No padding row is read into a result or written.  128 experts of 2048 x 768 with 4 rows each: GEMM1 141 us
// (805 MB of weights: 5.7 TB/s), GEMM2 71 (5.7 TB/s); with token rows in tiles of 256 on the M side they took 203 and 124.  Four 48 KB
// stages keep 128 KB of weights in flight per SM; pairing SMs would halve the token bytes only, which are few.
//
//   kFwd1    act = SwiGLU(X W1^T)   gate block + up block of a tile
//   kFwd2    y = act W2^T, rows scattered to their sources
//
// Warps as in grouped_gemm.cu: 0 TMA producer, 1 tensor memory + MMA issue, 2-9 epilogue, 10-11 transport (kComm).
// Every mbarrier wait is bounded; on a timeout the CTA raises its abort flag, records a status, lets issued copies
// land, frees its tensor memory and returns.
#include "narrow_gemm.h"

#include <cuda_bf16.h>

#include "comm.cuh"
#include "common.cuh"
#include "tcgen05.cuh"

namespace epb {
namespace {

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int NT = 128;                                   // most token rows of a tile
constexpr int BOX_N = kNarrowBoxRows;                     // token rows of one TMA box
constexpr int A_BYTES = 2 * BM * BK * 2;                  // two 128-row weight blocks
constexpr int STAGE_BYTES = A_BYTES + NT * BK * 2;        // 48 KB
constexpr int TMEM_COLS = 512;                            // 2 accumulator buffers x 2 weight blocks x NT columns
constexpr int NUM_THREADS = 320, COMM_WARPS = 2;
constexpr int COMM_SLOTS = 8;
constexpr int MAX_GROUPS = 320;
constexpr int kCtrlBytes = 1536;
constexpr int kStageHalfBytes = 32 * BM * 2;              // staging of four epilogue warps: 32 token rows x 128 features
template <int kComm>
constexpr int stages() { return kComm ? 3 : 4; }          // the transport warps' rings take the fourth stage
static_assert((4 * 2 + 4) * 8 + 8 + (MAX_GROUPS + 1) * 4 <= kCtrlBytes, "control block does not fit");

struct Tile {
  int g, mt;
  int row, n;      // first buffer row and real rows (<= NT)
  int wslot;
};

// Token tiles of a group: as few as NT allows, all of nearly the same size (multiples of BOX_N).
__device__ __forceinline__ int tiles_of(int rows) { return ceil_div(rows, NT); }

// `g` is the caller's cursor: tile indices only grow, so the walk over the prefix continues where it stopped.
__device__ __forceinline__ bool find_tile(const GemmArgs& a, int n_groups, const int* tile_prefix, int t, int& g, Tile& out) {
  while (g < n_groups && t >= tile_prefix[g + 1]) ++g;
  if (g >= n_groups) return false;
  const int rows = a.group_rows[g];
  const int nt_count = tiles_of(rows);
  const int local = t - tile_prefix[g];
  out.g = g;
  out.mt = local / nt_count;                 // token tiles of one weight tile are neighbours: they share it through L2
  const int nt = local - out.mt * nt_count;
  const int per = round_up(ceil_div(rows, nt_count), BOX_N);
  out.row = a.group_off[g] + nt * per;
  out.n = max(0, min(per, rows - nt * per));
  out.wslot = a.group_wslot[g];
  return true;
}

// Write 32 token rows x 128 features (256 B per row) staged by the four warps of a half: two rows per instruction.
// `mine` is where the lane's own token's features go (null: not stored); lane = token of the chunk, the same in all four warps.
__device__ __forceinline__ void flush_rows(const uint4* tile, int quarter, int lane, char* mine, int pieces) {
  const unsigned long long p = reinterpret_cast<unsigned long long>(mine);
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int tok = quarter * 8 + it * 2 + (lane >> 4), piece = lane & 15;
    const unsigned long long base = __shfl_sync(0xffffffffu, p, tok);
    if (base != 0ull && piece < pieces) *reinterpret_cast<uint4*>(base + piece * 16) = tile[tok * 16 + piece];
  }
}
// Stage one value per (token, feature): lane = feature, element j = token.  A warp writes 64 contiguous bytes per token.
template <typename F>
__device__ __forceinline__ void stage_and_flush(__nv_bfloat16* stg, int half, int quarter, int lane, char* mine, int pieces, F value) {
  half_sync(half);  // the previous flush has read the tile
#pragma unroll
  for (int j = 0; j < 32; ++j) stg[j * BM + quarter * 32 + lane] = value(j);
  half_sync(half);
  flush_rows(reinterpret_cast<const uint4*>(stg), quarter, lane, mine, pieces);
}

template <int kMode, int kComm>
__global__ void __launch_bounds__(NUM_THREADS + (kComm ? COMM_WARPS * 32 : 0), 1)
narrow_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   const __grid_constant__ GemmArgs args) {
  constexpr int STAGES = stages<kComm>();

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;       // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* tile_prefix = abort_flag + 1;        // [MAX_GROUPS + 1]
  uint8_t* stage_tiles = smem + STAGES * STAGE_BYTES + kCtrlBytes;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_groups = min(args.totals[1], args.n_groups_cap);
  const int m_tiles = kMode == kFwd1 ? args.N / BM : ceil_div(args.N, 2 * BM);
  const int kblocks = args.K / BK;

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
    warp_tile_prefix(tile_prefix, n_groups, lane, [&](int g) { return tiles_of(args.group_rows[g]) * m_tiles; });
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int total_tiles = tile_prefix[n_groups];
  volatile int* abort_v = abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    int stage = 0, cursor = 0;
    uint32_t phase = 0;
    Tile t;
    const unsigned long long wait_ns = args.wait_ns ? args.wait_ns : kWaitBudgetNs;
    int seen_row_tile = -1, seen_slot = -1;  // waits already satisfied (rows and slots only grow along the tile list)
    if (lane == 0) {
      bool go = true;
      for (int ti = blockIdx.x; ti < total_tiles && go; ti += gridDim.x) {
        if (*abort_v || !find_tile(args, n_groups, tile_prefix, ti, cursor, t)) break;
        const bool two = kMode == kFwd1 || t.mt * 2 * BM + BM < args.N;   // the second weight block exists
        const int boxes = ceil_div(t.n, BOX_N);
        // replica weights first: only the first loads of a tile wait for the rows as well
        if (args.pull_cnt != nullptr && t.wslot >= args.home_cap && t.wslot != seen_slot) {
          if (!flag_wait<false>(args.pull_cnt + (t.wslot - args.home_cap), args.pull_expected, wait_ns, abort_v, args.status, 6, t.wslot)) break;
          seen_slot = t.wslot;
        }
        if (args.arrive != nullptr && t.n > 0) {
          const int last = min(t.row + t.n - 1, args.row_capacity - 1) / args.arrive_tile_rows;
          for (int i = t.row / args.arrive_tile_rows; i <= last && go; ++i) {
            if (i == seen_row_tile) continue;
            if (!flag_wait<true>(args.arrive + i, args.arrive_expected, wait_ns, abort_v, args.status, 5, i)) go = false;
            else seen_row_tile = i;
          }
          if (!go) break;
        }
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_v, args.status, 1)) {
            go = false;
            break;
          }
          uint8_t* sA = tiles + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          uint64_t* fb = &full_bar[stage];
          mbar_expect_tx(fb, (two ? A_BYTES : A_BYTES / 2) + boxes * BOX_N * BK * 2);
          const int m0 = kMode == kFwd1 ? t.mt * BM : t.mt * 2 * BM;
          const int m1 = kMode == kFwd1 ? args.N + t.mt * BM : m0 + BM;
          tma_load_3d(sA, &tmW, fb, kb * BK, m0, t.wslot);
          if (two) tma_load_3d(sA + A_BYTES / 2, &tmW, fb, kb * BK, m1, t.wslot);
          for (int j = 0; j < boxes; ++j) tma_load_2d(sB + j * BOX_N * BK * 2, &tmX, fb, kb * BK, t.row + j * BOX_N);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int stage = 0, cursor = 0, local = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      Tile t;
      for (int ti = blockIdx.x; ti < total_tiles && !*abort_v; ti += gridDim.x, ++local) {
        if (!find_tile(args, n_groups, tile_prefix, ti, cursor, t)) break;
        const bool two = kMode == kFwd1 || t.mt * 2 * BM + BM < args.N;
        const int buf = local & 1;
        if (!mbar_wait(&acc_empty[buf], acc_phase[buf] ^ 1u, abort_v, args.status, 2)) break;
        acc_phase[buf] ^= 1u;
        tc_fence_after();
        const uint32_t d0 = tmem_base + (uint32_t)(buf * 2 * NT), d1 = d0 + NT;
        const uint32_t idesc = make_idesc(false, false, max(16, round_up(t.n, 16)), BM);
        if (args.trace != nullptr && local == 0) {
          // profiling aid: when did the first tile of the launch have its operands? (the wait repeats below)
          if (mbar_wait(&full_bar[stage], phase, abort_v, args.status, 3)) atomicMin(args.trace + 3, globaltimer_ns());
        }
        bool failed = false;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_v, args.status, 3)) {
            failed = true;
            break;
          }
          tc_fence_after();
          const uint32_t sA = smem_u32(tiles + stage * STAGE_BYTES), sB = sA + A_BYTES;
          const uint64_t da = make_desc(sA, 16, 1024), db = make_desc(sB, 16, 1024);
          constexpr uint32_t k_step = (UMMA_K * 2) >> 4;
          constexpr uint32_t a_block = (A_BYTES / 2) >> 4;   // second weight block of the stage
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint32_t acc = (kb | k) ? 1u : 0u;
            umma_bf16(d0, da + (uint64_t)(k * k_step), db + (uint64_t)(k * k_step), idesc, acc);
            if (two) umma_bf16(d1, da + (uint64_t)(a_block + k * k_step), db + (uint64_t)(k * k_step), idesc, acc);
          }
          umma_commit(&empty_bar[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (failed) break;
        if (args.trace != nullptr) atomicMax(args.trace + 2, globaltimer_ns());
        umma_commit(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else if (kComm != 0 && warp >= NUM_THREADS / 32) {
    // ------------------------------------------------------------ transport (warps 10, 11)
    const int w = warp - NUM_THREADS / 32;
    if (args.trace != nullptr && lane == 0) atomicMin(args.trace, globaltimer_ns());
    comm_run<COMM_SLOTS>(args.comm, (int)blockIdx.x * COMM_WARPS + w, (int)gridDim.x * COMM_WARPS,
                         stage_tiles + 2 * kStageHalfBytes + w * comm_warp_bytes<COMM_SLOTS>(), args.status,
                         args.trace != nullptr ? args.trace + 8 : nullptr);
    if (args.trace != nullptr && lane == 0) atomicMax(args.trace + 1, globaltimer_ns());
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    // Lane = output feature (TMEM lane), column = token.  Four warps (one half) cover 128 features; kFwd1 splits a tile's
    // 32-token chunks between the halves (each needs gate and up of its tokens), the plain modes give each half one
    // weight block.  The halves transpose through shared memory and store 256 contiguous bytes per token row.
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    __nv_bfloat16* stg = reinterpret_cast<__nv_bfloat16*>(stage_tiles + half * kStageHalfBytes);
    uint32_t acc_phase[2] = {0, 0};
    int local = 0, cursor = 0;
    Tile t;
    char* out0 = reinterpret_cast<char*>(args.out0);
    char* out1 = reinterpret_cast<char*>(args.out1);
    for (int ti = blockIdx.x; ti < total_tiles; ti += gridDim.x, ++local) {
      if (!find_tile(args, n_groups, tile_prefix, ti, cursor, t)) break;
      const int buf = local & 1;
      // the abort flag may be seen by some warps of a half only; a half must leave together (it shares barriers)
      const bool ok = mbar_wait(&acc_full[buf], acc_phase[buf], abort_v, args.status, 4);
      if (!half_all(half, ok)) break;
      acc_phase[buf] ^= 1u;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 2 * NT);
      const int chunks = ceil_div(t.n, 32);
      if (kMode == kFwd1) {
        const int F = args.N;
        for (int c = half; c < chunks; c += 2) {
          const int tok = c * 32 + lane;
          const size_t row = (size_t)t.row + tok;
          const bool real = tok < t.n && row < (size_t)args.row_capacity;
          char* arow = real ? out1 + (row * (size_t)F + t.mt * BM) * 2 : nullptr;
          const float my_scale = (real && args.row_scale != nullptr) ? __ldcg(args.row_scale + row) : 1.f;
          uint32_t g[32], u[32];
          tmem_ld32(taddr + c * 32, g);
          tmem_ld32(taddr + NT + c * 32, u);
          tmem_ld_wait();
          stage_and_flush(stg, half, quarter, lane, arow, 16, [&](int j) {
            // activation from the bf16-rounded pre-activations, exactly as the wide kernel computes it
            const float gr = __bfloat162float(__float2bfloat16_rn(__uint_as_float(g[j])));
            const float ur = __bfloat162float(__float2bfloat16_rn(__uint_as_float(u[j])));
            const float rs = __shfl_sync(0xffffffffu, my_scale, j);
            return __float2bfloat16_rn(rs * gr * sigmoidf_fast(gr) * ur);
          });
        }
      } else {
        const int col0 = t.mt * 2 * BM + half * BM;                          // first feature of this half's weight block
        const int pieces = min(16, (args.N - col0) / 8);                     // 16-byte pieces of a row that exist
        for (int c = 0; c < chunks && pieces > 0; ++c) {
          const int tok = c * 32 + lane;
          const size_t row = (size_t)t.row + tok;
          char* orow = nullptr;
          if (tok < t.n && row < (size_t)args.row_capacity) {
            if (args.meta != nullptr) {
              const int2 mt = args.meta[row];
              char* base = args.out_ptrs ? reinterpret_cast<char*>(args.out_ptrs[mt.x]) : out0;
              orow = base + ((size_t)mt.y * args.N + col0) * 2;
            } else {
              orow = out0 + (row * (size_t)args.N + col0) * 2;
            }
          }
          uint32_t v[32];
          tmem_ld32(taddr + half * NT + c * 32, v);
          tmem_ld_wait();
          stage_and_flush(stg, half, quarter, lane, orow, pieces, [&](int j) { return __float2bfloat16_rn(__uint_as_float(v[j])); });
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    if (args.done_ctr != nullptr) __threadfence_system();  // this warp's (peer) stores before the completion signal
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (args.done_ctr != nullptr && threadIdx.x == 0) signal_launch_done(args);
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

template <int kComm>
constexpr size_t smem_bytes() {
  return stages<kComm>() * STAGE_BYTES + 1024 /*align*/ + kCtrlBytes + 2 * kStageHalfBytes +
         (kComm ? COMM_WARPS * comm_warp_bytes<COMM_SLOTS>() : 0);
}
static_assert(smem_bytes<0>() <= 232448 && smem_bytes<1>() <= 232448, "shared memory budget");

template <int kMode, int kComm>
cudaError_t launch_mode(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms, cudaStream_t stream) {
  static bool configured[kMaxTrackedDevices] = {};
  constexpr size_t smem = smem_bytes<kComm>();
  int dev;
  if (device_needs_setup(configured, &dev)) {
    cudaError_t e = cudaFuncSetAttribute(narrow_gemm_kernel<kMode, kComm>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    device_setup_done(configured, dev);
  }
  narrow_gemm_kernel<kMode, kComm><<<num_sms, NUM_THREADS + (kComm ? COMM_WARPS * 32 : 0), smem, stream>>>(tmW, tmX, args);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_narrow_gemm(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms,
                               cudaStream_t stream) {
  if (args.n_groups_cap > MAX_GROUPS || args.K <= 0 || args.K % BK != 0 || args.N % 32 != 0) return cudaErrorInvalidValue;
  if (args.arrive != nullptr && args.arrive_tile_rows <= 0) return cudaErrorInvalidValue;
  if (args.mode == kFwd1 && (args.N % BM != 0 || args.out0 != nullptr)) return cudaErrorInvalidValue;
  const bool comm = args.comm.do_dispatch || args.comm.do_pad || args.comm.do_pull;
  switch (args.mode) {
    case kFwd1: return comm ? launch_mode<kFwd1, 1>(tmW, tmX, args, num_sms, stream) : launch_mode<kFwd1, 0>(tmW, tmX, args, num_sms, stream);
    case kFwd2:
      if (comm) return cudaErrorInvalidValue;
      return launch_mode<kFwd2, 0>(tmW, tmX, args, num_sms, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace epb
