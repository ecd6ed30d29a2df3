// Grouped GEMM of token rows for sm_100a: a CTA pair (tcgen05.mma.cta_group::2) holds 256 WEIGHT rows (output features) as the
// M operand and up to 256 token rows as its N columns.
//
// The rows of a group are ragged.  With token rows on the M side a group costs whole tiles of 256 rows, 128 rows of padding a
// group on average; as N columns they are rounded up to 32, and a group is cut into as few tiles as 256 columns allow, of
// nearly the same size.  No padding row is read into a result.  Against the same ring and tile size with token rows on the M
// side, in long runs (where the power limit sets the clock): 64 experts of 2048 x 1408, 49153 rows that 256-row tiles pad by
// 18 %: GEMM1 511-539 -> 494-514 us, GEMM2 259-277 -> 245-262, Dgrad2 276-295 -> 260-280, Dgrad1 480-508 -> 447-479; 12245 rows
// on 64 experts of 2048 x 1024 (padded by 53 %; reading the weights is half the time) 2-7 % less; nothing to save without padding.
//
//   kFwd1    h = X W1^T, act = SwiGLU(h)   a tile is 128 features: each CTA holds 64 gate and their 64 up rows
//   kFwd2    y = act W2^T, rows scattered to their sources            (weights K-major)
//   kDgrad1  dX = dH W1 (scattered) or dAct = dY W2 (local rows)      (weights MN-major)
//   kPlain   C = A B^T, rows kept local
//
// Warps as in grouped_gemm.cu: 0 TMA producer, 1 tensor memory + MMA issue, 2-9 epilogue, 10-11 transport (kComm).
// Every mbarrier wait is bounded; on a timeout the CTA raises its abort flag, records a status, lets issued copies
// land, frees its tensor memory and returns.
#include "ragged_gemm.h"

#include <cuda_bf16.h>

#include "comm.cuh"
#include "common.cuh"
#include "tcgen05.cuh"

namespace epb {
namespace {

constexpr int BM = 128, BK = 64, UMMA_K = 16;      // BM: weight rows of one CTA
constexpr int NT = 256;                            // most token columns of a tile
// One k-block: 16 KB of weights and 16 KB of token rows, one copy each.  A CTA's token box is always NT / 2 = 128 rows: what a
// smaller tile reads past its rows is never used.  (Boxes of 32 rows, only as many as needed, made the launches 5-12 % slower.)
constexpr int A_BYTES = BM * BK * 2, SUB_BYTES = A_BYTES + NT / 2 * BK * 2;
constexpr int TMEM_COLS = 512;                     // two accumulators of NT columns
constexpr int NUM_THREADS = 320, COMM_WARPS = 2;
constexpr int COMM_SLOTS = 8;
constexpr int MAX_GROUPS = 320;
constexpr int kCtrlBytes = 1536;
constexpr int kStageBytes = 32 * BM * 2;           // 32 tokens x 128 features; two per half of the epilogue warps

// Ring: without transport three stages of two k-blocks, with it four of one.  Every tcgen05.commit leaves the tensor pipe idle
// for some 45 cycles, and a k-block is only 512 cycles of MMAs: with two commits a k-block (one per CTA of the pair) the pipe was
// at most 78 % busy with no loads and no epilogue at all, with one multicast commit 84 %, with one per two k-blocks 96 %.
template <int kComm>
struct Ring {
  static constexpr int kSub = kComm ? 1 : 2;
  static constexpr int STAGES = kComm ? 4 : 3;
  static constexpr int STAGE_BYTES = kSub * SUB_BYTES;
};
static_assert((6 * 2 + 4) * 8 + 8 + (MAX_GROUPS + 1) * 4 <= kCtrlBytes, "control block does not fit");

struct Tile {
  int wt;        // weight tile
  int row, n;    // first buffer row and real rows
  int cols;      // n rounded up to 32: columns of the MMA
  int pad;       // rows of zeros that kFwd1 writes after the n real ones (last tile of a group; else 0)
  int wslot;
};

// Tile t of the list; `g` is the caller's cursor (0 before its first tile): tile indices only grow.  The weight tiles of one
// token tile are neighbours (they share its rows through L2).
__device__ __forceinline__ bool find_tile(const GemmArgs& a, int n_groups, int m_tiles, const int* tile_prefix, int t, int& g, Tile& out) {
  while (g < n_groups && t >= tile_prefix[g + 1]) ++g;
  if (g >= n_groups) return false;
  const int rows = a.group_rows[g];
  const int local = t - tile_prefix[g];
  const int tt = local / m_tiles, count = ceil_div(rows, NT);
  const int per = round_up(ceil_div(rows, count), 32);
  out.wt = local - tt * m_tiles;
  out.row = a.group_off[g] + tt * per;
  out.n = min(per, rows - tt * per);
  out.cols = round_up(out.n, 32);
  out.pad = tt == count - 1 ? round_up(rows, a.pad_rows > 0 ? a.pad_rows : NT) - rows : 0;
  out.wslot = a.group_wslot[g];
  return true;
}

// Accumulator columns [0, 32) of 16 TMEM lanes.  Thread t gets, for each group i of 8 columns, lane t / 4 (registers 4i, 4i + 1)
// and lane t / 4 + 8 (4i + 2, 4i + 3) of columns 8i + 2 (t % 4) and the one after: 8 x 8 fragments.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void stmatrix_t(uint32_t saddr, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(m0), "r"(m1), "r"(m2), "r"(m3)
               : "memory");
}
// Staging: 16-byte piece p (8 features) of token r lives at index r * 16 + (p ^ (r & 7)): the eight tokens of a transposed 8 x 8
// matrix and the pieces of one token both fall into different banks.
__device__ __forceinline__ int piece_index(int r, int p) { return r * 16 + (p ^ (r & 7)); }

// This warp's 32 features (TMEM lanes) of 32 tokens, rounded to bf16, into the staging tile, token by token.  Two loads and four
// stores of 8 x 8 matrices, which transpose on the way: one 16-bit store per token took 32.
__device__ __forceinline__ void stage_chunk(uint32_t taddr, uint4* tile, int quarter, int lane) {
  uint32_t r[2][16];
  tmem_ld_16x32(taddr, r[0]);
  tmem_ld_16x32(taddr + (16u << 16), r[1]);
  tmem_ld_wait();
  const int tok = ((lane >> 4) << 3) + (lane & 7), hi = (lane >> 3) & 1;  // the staging row whose address this lane gives
#pragma unroll
  for (int lh = 0; lh < 2; ++lh)
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      uint32_t m[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)  // {first 8 features, next 8} of token group i, then of i + 1
        m[k] = pack_bf16(__uint_as_float(r[lh][4 * (i + (k >> 1)) + 2 * (k & 1)]), __uint_as_float(r[lh][4 * (i + (k >> 1)) + 2 * (k & 1) + 1]));
      stmatrix_t(smem_u32(tile + piece_index(8 * i + tok, quarter * 4 + lh * 2 + hi)), m[0], m[1], m[2], m[3]);
    }
}

template <int kMode, int kComm>
__global__ void __launch_bounds__(NUM_THREADS + (kComm ? COMM_WARPS * 32 : 0), 1)
ragged_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   const __grid_constant__ GemmArgs args) {
  using G = Ring<kComm>;
  constexpr int STAGES = G::STAGES, STAGE_BYTES = G::STAGE_BYTES, kSub = G::kSub;
  constexpr bool kWMn = kMode == kDgrad1;
  constexpr int kFeatures = kMode == kFwd1 ? 128 : 256;  // output columns of a tile

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
  const int cta_rank = (int)cluster_ctarank();  // rank 0 of the pair issues the MMAs
  const int tile_first = blockIdx.x / 2, tile_stride = gridDim.x / 2;
  const int n_groups = min(args.totals[1], args.n_groups_cap);
  const int m_tiles = ceil_div(args.N, kFeatures);
  const int kblocks = ceil_div(args.K, BK);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 16);  // 8 epilogue warps of each CTA
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, TMEM_COLS);
  if (warp == 2)
    warp_tile_prefix(tile_prefix, n_groups, lane, [&](int g) { return ceil_div(args.group_rows[g], NT) * m_tiles; });
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  volatile int* abort_v = abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0, cursor = 0;
      uint32_t phase = 0;
      Tile t, next;
      bool have = find_tile(args, n_groups, m_tiles, tile_prefix, tile_first, cursor, t), go = true;
      const unsigned long long wait_ns = args.wait_ns ? args.wait_ns : kWaitBudgetNs;
      int seen_row_tile = -1, seen_slot = -1;  // waits already satisfied (rows and slots only grow along the tile list)
      for (int ti = tile_first; have && go && !*abort_v; ti += tile_stride, t = next) {
        have = find_tile(args, n_groups, m_tiles, tile_prefix, ti + tile_stride, cursor, next);
        if (args.arrive != nullptr) {
          // rows of this tile must have arrived from every sender
          const int last = min(t.row + t.n - 1, args.row_capacity - 1) / args.arrive_tile_rows;
          for (int i = t.row / args.arrive_tile_rows; i <= last && go; ++i) {
            if (i == seen_row_tile) continue;
            if (!flag_wait<true>(args.arrive + i, args.arrive_expected, wait_ns, abort_v, args.status, 5, i)) go = false;
            else seen_row_tile = i;
          }
          if (!go) break;
        }
        if (args.pull_cnt != nullptr && t.wslot >= args.home_cap && t.wslot != seen_slot) {
          if (!flag_wait<false>(args.pull_cnt + (t.wslot - args.home_cap), args.pull_expected, wait_ns, abort_v, args.status, 6, t.wslot)) break;
          seen_slot = t.wslot;
        }
        const int x_row = t.row + cta_rank * (t.cols / 2);      // this CTA's half of the token columns
        const int m_off = t.wt * kFeatures + cta_rank * (kFeatures / 2);
        for (int kb0 = 0; kb0 < kblocks; kb0 += kSub) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_v, args.status, 1)) {
            go = false;
            break;
          }
          uint64_t* fb = &full_bar[stage];
          const int subs = min(kSub, kblocks - kb0);
          if (cta_rank == 0) mbar_expect_tx(fb, 2 * subs * SUB_BYTES);  // both CTAs' bytes land on the leader's barrier
          for (int sub = 0; sub < subs; ++sub) {
            const int k0 = (kb0 + sub) * BK;
            uint8_t* sA = tiles + stage * STAGE_BYTES + sub * SUB_BYTES;
            uint8_t* sB = sA + A_BYTES;
            if (kMode == kFwd1) {
              tma_load_4d_pair(sA, &tmW, fb, k0, m_off, 0, t.wslot);
            } else if (kWMn) {
              tma_load_4d_pair(sA, &tmW, fb, 0, k0, m_off / 64, t.wslot);
            } else {
              tma_load_3d_pair(sA, &tmW, fb, k0, m_off, t.wslot);
            }
            tma_load_2d_pair(sB, &tmX, fb, k0, x_row);
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
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (lane == 0 && cta_rank == 0) {
      int stage = 0, cursor = 0, local = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      Tile t, next;
      bool have = find_tile(args, n_groups, m_tiles, tile_prefix, tile_first, cursor, t);
      for (int ti = tile_first; have && !*abort_v; ti += tile_stride, ++local, t = next) {
        have = find_tile(args, n_groups, m_tiles, tile_prefix, ti + tile_stride, cursor, next);
        const int buf = local & 1;
        if (!mbar_wait(&acc_empty[buf], acc_phase[buf] ^ 1u, abort_v, args.status, 2)) break;
        acc_phase[buf] ^= 1u;
        tc_fence_after();
        if (args.trace != nullptr && local == 0) {
          // first operands of this CTA's first tile have landed?  (start of useful tensor work)
          if (mbar_wait(&full_bar[stage], phase, abort_v, args.status, 3)) atomicMin(args.trace + 3, globaltimer_ns());
        }
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * NT);
        const uint32_t idesc = make_idesc(kWMn, false, t.cols, 2 * BM);
        bool failed = false;
        for (int kb0 = 0; kb0 < kblocks; kb0 += kSub) {
          if (!mbar_wait(&full_bar[stage], phase, abort_v, args.status, 3)) {
            failed = true;
            break;
          }
          tc_fence_after();
          const int subs = min(kSub, kblocks - kb0);
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub) {
            if (sub >= subs) break;
            const uint32_t sA = smem_u32(tiles + stage * STAGE_BYTES + sub * SUB_BYTES), sB = sA + A_BYTES;
            const uint64_t da = kWMn ? make_desc(sA, 8192, 1024) : make_desc(sA, 16, 1024), db = make_desc(sB, 16, 1024);
            constexpr uint32_t a_step = kWMn ? (UMMA_K * 128) >> 4 : (UMMA_K * 2) >> 4, b_step = (UMMA_K * 2) >> 4;
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16_pair(tmem_d, da + (uint64_t)(k * a_step), db + (uint64_t)(k * b_step), idesc, (kb0 | sub | k) ? 1u : 0u);
          }
          umma_commit_both(&empty_bar[stage]);  // frees the stage in both CTAs once these MMAs have read it
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (failed) break;
        if (args.trace != nullptr) atomicMax(args.trace + 2, globaltimer_ns());
        umma_commit_both(&acc_full[buf]);  // accumulator ready for the epilogue warps of both CTAs
      }
    }
    __syncwarp();
  } else if (kComm != 0 && warp >= NUM_THREADS / 32) {
    // ------------------------------------------------------------ transport (warps 10, 11)
    const int w = warp - NUM_THREADS / 32;
    if (args.trace != nullptr && lane == 0) atomicMin(args.trace, globaltimer_ns());
    comm_run<COMM_SLOTS>(args.comm, (int)blockIdx.x * COMM_WARPS + w, (int)gridDim.x * COMM_WARPS,
                         stage_tiles + 4 * kStageBytes + w * comm_warp_bytes<COMM_SLOTS>(), args.status,
                         args.trace != nullptr ? args.trace + 8 : nullptr);
    if (args.trace != nullptr && lane == 0) atomicMax(args.trace + 1, globaltimer_ns());
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9 of both CTAs)
    // TMEM lane = output feature, column = token.  The four warps of a half cover the CTA's 128 features and take every other
    // 32-token chunk: they transpose it into a staging tile, meet, and write whole rows (128 or 256 contiguous bytes per token).
    // Two staging tiles a half, so that one meeting a chunk is enough: a warp that writes a tile again has met warps that were
    // done reading it.
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int tid = quarter * 32 + lane;
    uint4* stg = reinterpret_cast<uint4*>(stage_tiles + half * 2 * kStageBytes);
    uint32_t acc_phase[2] = {0, 0};
    int local = 0, cursor = 0, sbuf = 0;
    Tile t;
    char* out0 = reinterpret_cast<char*>(args.out0);
    char* out1 = reinterpret_cast<char*>(args.out1);
    for (int ti = tile_first; find_tile(args, n_groups, m_tiles, tile_prefix, ti, cursor, t); ti += tile_stride, ++local) {
      const int buf = local & 1;
      const int chunks = t.cols / 32;
      const int col0 = t.wt * kFeatures + cta_rank * (kFeatures / 2);  // this CTA's first output column
      // where the row of token `lane` of chunk c goes (null: nowhere)
      auto row_ptr = [&](int c) -> char* {
        const int tok = c * 32 + lane;
        const size_t row = (size_t)t.row + tok;
        if (tok >= t.n || row >= (size_t)args.row_capacity) return nullptr;
        if (args.meta == nullptr) return out0 + (row * (size_t)args.N + col0) * 2;
        const int2 mt = args.meta[row];
        char* base = args.out_ptrs ? reinterpret_cast<char*>(args.out_ptrs[mt.x]) : out0;
        return base + ((size_t)mt.y * args.N + col0) * 2;
      };
      auto row_scale = [&](int c) -> float {  // the gate weight of token `lane` of chunk c
        const int tok = c * 32 + lane;
        return tok < t.n && t.row + tok < args.row_capacity ? __ldcg(args.row_scale + t.row + tok) : 1.f;
      };
      // looked up while the tile is still being computed, then one chunk ahead (an earlier launch has stored the rows' sources)
      char* orow = kMode == kFwd1 ? nullptr : row_ptr(half);
      // the abort flag may be seen by some warps of a half only; a half must leave together (it shares barriers)
      const bool ok = mbar_wait(&acc_full[buf], acc_phase[buf], abort_v, args.status, 4);
      if (!half_all(half, ok)) break;
      acc_phase[buf] ^= 1u;
      tc_fence_after();
      // (the senders store the gate weights before the rows' arrival, which the producer has waited for)
      float rs = kMode == kFwd1 && args.row_scale != nullptr ? row_scale(half) : 1.f;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * NT);
      if (kMode == kFwd1) {
        const int F = args.N;
        // rows after the group's last one are written as zeros (Wgrad reads them), unless nothing is kept for a backward
        const int end = t.n + (out0 != nullptr ? t.pad : 0);
        for (int c = half; c * 32 < end; c += 2, sbuf ^= 1) {
          uint4* tile = stg + sbuf * (kStageBytes / 16);
          const float scale = rs;
          if (c < chunks) {
            stage_chunk(taddr + c * 32, tile, quarter, lane);
            if (args.row_scale != nullptr) rs = row_scale(c + 2);
          }
          half_sync(half);
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            const int tk = it * 16 + (tid >> 3), p = tid & 7, tok = c * 32 + tk;  // eight threads a token
            const size_t row = (size_t)t.row + tok;
            const float s = __shfl_sync(0xffffffffu, scale, tk);
            uint4 g = make_uint4(0, 0, 0, 0), u = g, act = g;
            if (tok < t.n) {
              g = tile[piece_index(tk, p)];
              u = tile[piece_index(tk, 8 + p)];
              const uint32_t* gw = reinterpret_cast<const uint32_t*>(&g);
              const uint32_t* uw = reinterpret_cast<const uint32_t*>(&u);
              uint32_t* aw = reinterpret_cast<uint32_t*>(&act);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                // activation from the bf16-rounded pre-activations, exactly what backward will read
                const float2 g2 = unpack_bf16(gw[k]), u2 = unpack_bf16(uw[k]);
                aw[k] = pack_bf16(s * g2.x * sigmoidf_fast(g2.x) * u2.x, s * g2.y * sigmoidf_fast(g2.y) * u2.y);
              }
            }
            if (tok < end && row < (size_t)args.row_capacity) {
              if (out0 != nullptr) {
                char* hrow = out0 + (row * (size_t)(2 * F) + col0) * 2 + p * 16;
                *reinterpret_cast<uint4*>(hrow) = g;
                *reinterpret_cast<uint4*>(hrow + (size_t)F * 2) = u;
              }
              *reinterpret_cast<uint4*>(out1 + (row * (size_t)F + col0) * 2 + p * 16) = act;
            }
          }
        }
      } else {
        const int pieces = min(16, (args.N - col0) / 8);  // 16-byte pieces of a row that exist (may be none)
        for (int c = half; c < chunks; c += 2, sbuf ^= 1) {
          uint4* tile = stg + sbuf * (kStageBytes / 16);
          const unsigned long long mine = reinterpret_cast<unsigned long long>(orow);
          stage_chunk(taddr + c * 32, tile, quarter, lane);
          orow = row_ptr(c + 2);
          half_sync(half);
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int tk = it * 8 + (tid >> 4), p = tid & 15;  // sixteen threads a token
            const unsigned long long base = __shfl_sync(0xffffffffu, mine, tk);
            if (base != 0ull && p < pieces) *reinterpret_cast<uint4*>(base + p * 16) = tile[piece_index(tk, p)];
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[buf]), 0));  // the leader's issuer may reuse the buffer
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
  cluster_sync_all();  // neither CTA leaves while the other may still signal it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <int kComm>
constexpr size_t smem_bytes() {
  return Ring<kComm>::STAGES * Ring<kComm>::STAGE_BYTES + 1024 /*align*/ + kCtrlBytes + 4 * kStageBytes +
         (kComm ? COMM_WARPS * comm_warp_bytes<COMM_SLOTS>() : 0);
}
static_assert(smem_bytes<0>() <= 232448 && smem_bytes<1>() <= 232448, "shared memory budget");

template <int kMode, int kComm>
cudaError_t launch_mode(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms, cudaStream_t stream) {
  static bool configured[kMaxTrackedDevices] = {};
  constexpr size_t smem = smem_bytes<kComm>();
  int dev;
  if (device_needs_setup(configured, &dev)) {
    cudaError_t e = cudaFuncSetAttribute(ragged_gemm_kernel<kMode, kComm>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    device_setup_done(configured, dev);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(num_sms / 2 * 2));
  cfg.blockDim = dim3(NUM_THREADS + (kComm ? COMM_WARPS * 32 : 0));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, ragged_gemm_kernel<kMode, kComm>, tmW, tmX, args);
}

}  // namespace

cudaError_t launch_ragged_gemm(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms,
                               cudaStream_t stream) {
  if (args.n_groups_cap > MAX_GROUPS || args.N % 32 != 0) return cudaErrorInvalidValue;
  if ((args.mode == kFwd1 && args.N % 128 != 0) || (args.mode == kDgrad1 && args.N % 64 != 0)) return cudaErrorInvalidValue;
  if (args.arrive != nullptr && args.arrive_tile_rows <= 0) return cudaErrorInvalidValue;
  const bool comm = args.comm.do_dispatch || args.comm.do_pad || args.comm.do_pull;
  switch (args.mode) {
    case kFwd1: return comm ? launch_mode<kFwd1, 1>(tmW, tmX, args, num_sms, stream) : launch_mode<kFwd1, 0>(tmW, tmX, args, num_sms, stream);
    case kDgrad1: return comm ? launch_mode<kDgrad1, 1>(tmW, tmX, args, num_sms, stream) : launch_mode<kDgrad1, 0>(tmW, tmX, args, num_sms, stream);
    case kFwd2: return comm ? cudaErrorInvalidValue : launch_mode<kFwd2, 0>(tmW, tmX, args, num_sms, stream);
    case kPlain: return comm ? cudaErrorInvalidValue : launch_mode<kPlain, 0>(tmW, tmX, args, num_sms, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace epb
