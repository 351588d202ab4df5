// The tcgen05 matrix product of gemm_tcgen05.cu: the kernel, templated on whether a block works alone or two blocks of a
// cluster work on one tile (cta_group::2), and its host-side launchers.
#pragma once

#include "qkv_rope.cuh"
#include "tcgen05.cuh"

namespace dl {

constexpr int T5_BM = 128;
constexpr int T5_BK = 64;                 // 64 bf16 = 128 bytes: one swizzle row
constexpr int T5_THREADS = 192;           // 6 warps
constexpr uint32_t T5_A_BYTES = T5_BM * T5_BK * 2;    // 16 KiB
constexpr uint32_t T5_STORE_BYTES = 4 * 32 * 128;     // per epilogue warp: 32 rows x 128 bytes of output, staged for coalesced stores

// A tile is 128 rows (256 for a pair of blocks, 128 each) by `bn` columns, a multiple of 32 up to 256, chosen per product
// (t5_launch). As many stages as fit: a stage is 128 rows of x and bn rows of W (bn / 2 for each block of a pair).
constexpr int T5_MAX_STAGES = 8;
constexpr uint32_t T5_TMEM_COLS = 512;                // two accumulators of up to 256 columns
constexpr uint32_t T5_BAR_BYTES = 256;
constexpr uint32_t T5_SMEM = 232448;                  // the 227 KiB a block may have
constexpr uint32_t T5_STAGE_ROOM = T5_SMEM - T5_STORE_BYTES - 1024 /* alignment */ - T5_BAR_BYTES;
__host__ __device__ constexpr uint32_t t5_stage_bytes(int bn, int cluster) { return T5_A_BYTES + bn / cluster * T5_BK * 2; }
__host__ __device__ constexpr int t5_stages(int bn, int cluster) {
  return T5_STAGE_ROOM / t5_stage_bytes(bn, cluster) < T5_MAX_STAGES ? T5_STAGE_ROOM / t5_stage_bytes(bn, cluster) : T5_MAX_STAGES;
}

enum { T5_OUT_BF16 = 0, T5_OUT_F32 = 1, T5_OUT_SWIGLU = 2, T5_OUT_QKV_ROPE = 3, T5_OUT_RELU2 = 4, T5_OUT_GELU = 5, T5_OUT_PAIRS = 6, T5_OUT_XIELU = 7 };
enum { T5_ERR_PRODUCER = 1, T5_ERR_MMA = 2, T5_ERR_EPILOGUE = 3 };

// Which output tile a tile number stands for. Tiles are numbered in groups of `group_m` row blocks: inside a
// group the row block changes fastest, then the column block; the groups follow one another. The blocks of the grid
// work on consecutive numbers at any time, so together they hold group_m row blocks of x and gridDim.x / group_m
// column blocks of W: both stay in L2 while they are used, and over the whole product W comes from memory once
// per group and x once. (Numbered along the columns first, as this kernel did at first, every row block brings all
// of W in again: with the 235 MB of a 4096 -> 2 x 14336 gate|up matrix that bound the product to memory, 1,684 us
// for 8,192 rows where the arithmetic needs 1,300.)
__host__ __device__ __forceinline__ void t5_tile_coords(int tile, int tiles_n, int num_tiles, int group_m, int* m_tile, int* n_tile) {
  const int tiles_m = num_tiles / tiles_n;
  const int per_group = group_m * tiles_n;
  const int g = tile / per_group;
  const int first_m = g * group_m;
  const int rows = group_m < tiles_m - first_m ? group_m : tiles_m - first_m;
  const int r = tile - g * per_group;
  *m_tile = first_m + r % rows;
  *n_tile = r / rows;
}

// gate_rows: for SwiGLU the number of gate features F (W has 2F rows); the tile's W rows are
// [n0, n0 + 128) and [F + n0, F + n0 + 128). Otherwise unused.
//
// The kernel is persistent: gridDim.x blocks (at most one per SM) walk the output tiles in the order
// tile = blockIdx.x, blockIdx.x + gridDim.x, ...; see t5_tile_coords for which tile a number stands for.
// The accumulator is double-buffered in tensor memory (2 x 256 columns): the epilogue warps drain
// one tile while the MMA warp fills the next.
//
// PAIR: the two blocks of a thread-block cluster compute one tile of 256 rows: each loads its own 128 rows of x and one half
// of the tile's W (for SwiGLU one the gate rows, the other the up rows), and the first block's tensor core instructions
// (cta_group::2) read both blocks' shared memory and write both blocks' tensor memory, 128 rows each. An SM so takes in
// 128 + bn / 2 rows a slice where a block alone takes in 128 + bn: the product is bound by that traffic from L2. The copies
// of both blocks count on the first block's "full" barrier (it expects the bytes of both); its commits arrive on the
// "empty" and "accumulator full" barriers of both; both blocks' epilogues arrive on its "accumulator empty" barrier.
// A grouped product: the rows of x come in runs, each run multiplied by a matrix of its own (the experts of a mixture),
// and which rows form a run is known on the device only. `tiles` lists row tiles as (matrix, first row, rows <= 128),
// `n_tiles[0]` says how many; matrix g lies w_rows rows below the first in the tensor map of W. A row tile may start at
// any row; the rows it holds past its run are multiplied with the wrong matrix and never stored. tiles == nullptr: a
// plain product. The list is written by a kernel in front, so a grouped product asks for nothing before its wait.
struct T5Groups {
  const int* tiles;
  const int* n_tiles;
  int w_rows;
};

template <bool PAIR>
__global__ void __launch_bounds__(T5_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    void* __restrict__ y, int ldy, int M, int N, int K, int mode, float out_scale, int gate_rows,
                    int tiles_n, int num_tiles_plain, int group_m, int* __restrict__ status, const QkvRope rope,
                    const T5Groups groups, const float* __restrict__ coeffs, const int bn) {
  constexpr int CLUSTER = PAIR ? 2 : 1;
  const int stages = t5_stages(bn, CLUSTER);
  const uint32_t stage_bytes = t5_stage_bytes(bn, CLUSTER);
  extern __shared__ unsigned char t5_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(t5_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* store_stage = tiles + static_cast<size_t>(stages) * stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(store_stage + T5_STORE_BYTES);
  uint64_t* full_bar = bars;                        // [stages] stage loaded (a pair: the first block's)
  uint64_t* empty_bar = bars + T5_MAX_STAGES;       // [stages] stage consumed
  uint64_t* acc_full = bars + 2 * T5_MAX_STAGES;        // [2] accumulator complete
  uint64_t* acc_empty = bars + 2 * T5_MAX_STAGES + 2;   // [2] accumulator drained (a pair: the first block's)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * T5_MAX_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = PAIR ? static_cast<int>(cluster_rank()) : 0;
  const int first_tile = static_cast<int>(blockIdx.x) / CLUSTER, tile_step = static_cast<int>(gridDim.x) / CLUSTER;
  const bool swiglu = mode == T5_OUT_SWIGLU;
  const int n_per_tile = swiglu ? bn / 2 : bn;            // output features per tile
  const int k_tiles = (K + T5_BK - 1) / T5_BK;
  const bool grouped = groups.tiles != nullptr;
  // (first row, first feature, first row of W's matrix, one past the last row to store) of a tile
  auto coords = [&](int tile, int num_tiles, int* m0, int* n0, int* w0, int* m_end) {
    if (grouped) {
      const int* g = groups.tiles + 3 * (tile / tiles_n);
      *m0 = g[1];
      *m_end = g[1] + g[2];
      *n0 = (tile % tiles_n) * n_per_tile;
      *w0 = g[0] * groups.w_rows;
    } else {
      int m_tile, n_tile;
      t5_tile_coords(tile, tiles_n, num_tiles, group_m, &m_tile, &n_tile);
      *m0 = (m_tile * CLUSTER + rank) * T5_BM;
      *n0 = n_tile * n_per_tile;
      *w0 = 0;
      *m_end = M;
    }
  };

  if (threadIdx.x == 0) {
    prefetch_tensor_map(&map_x);
    prefetch_tensor_map(&map_w);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4 * CLUSTER);        // one arrival per epilogue warp
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T5_TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T5_TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  if constexpr (PAIR) cluster_sync_all();              // both blocks' barriers exist before anything is sent to them

  if (warp == 0) {
    // TMA producer: the whole warp runs the loop (every lane polls the barrier), one elected lane issues the copies
    // The first stages' slices of W are requested before the wait on the kernel in front (programmatic dependent
    // launch): W does not depend on it. x, which does, follows after the wait.
    const uint32_t full0 = PAIR ? in_first_block(smem_u32(full_bar)) : smem_u32(full_bar);
    auto load_w = [&](int s, int kt, int n0) {
      unsigned char* b_dst = tiles + static_cast<size_t>(s) * stage_bytes + T5_A_BYTES;
      const int second_half = swiglu ? gate_rows + n0 : n0 + bn / 2;      // W row of the tile's second half
      if constexpr (PAIR) {
        tma_load_2d_pair(b_dst, &map_w, kt * T5_BK, rank == 0 ? n0 : second_half, full0 + s * 8);
      } else {
        tma_load_2d(b_dst, &map_w, kt * T5_BK, n0, &full_bar[s]);
        tma_load_2d(b_dst + bn / 2 * (T5_BK * 2), &map_w, kt * T5_BK, second_half, &full_bar[s]);
      }
    };
    auto load_x = [&](int s, int kt, int m0) {
      unsigned char* a_dst = tiles + static_cast<size_t>(s) * stage_bytes;
      if constexpr (PAIR) tma_load_2d_pair(a_dst, &map_x, kt * T5_BK, m0, full0 + s * 8);
      else tma_load_2d(a_dst, &map_x, kt * T5_BK, m0, &full_bar[s]);
    };
    // the first block of a pair expects the bytes of both
    auto expect = [&](int s) {
      if (rank == 0) mbar_expect_tx(&full_bar[s], CLUSTER * stage_bytes);
    };
    const int ahead = (!grouped && first_tile < num_tiles_plain) ? min(k_tiles, stages) : 0;
    if (ahead > 0) {
      int m0, n0, w0, m_end;
      coords(first_tile, num_tiles_plain, &m0, &n0, &w0, &m_end);
      if (elect_one()) {
        for (int kt = 0; kt < ahead; ++kt) {
          expect(kt);
          load_w(kt, kt, n0);
        }
      }
      __syncwarp();
      pdl_wait();
      pdl_trigger();
      if (elect_one()) {
        for (int kt = 0; kt < ahead; ++kt) load_x(kt, kt, m0);
      }
      __syncwarp();
    } else {
      pdl_wait();
      pdl_trigger();
    }
    const int num_tiles = grouped ? groups.n_tiles[0] * tiles_n : num_tiles_plain;      // (after the wait)
    int s = ahead % stages, round = ahead / stages;      // the next slice's stage, and how often the stages have gone round
    bool ok = true;
    for (int tile = first_tile; tile < num_tiles && ok; tile += tile_step) {
      int m0, n0, w0, m_end;
      coords(tile, num_tiles, &m0, &n0, &w0, &m_end);
      n0 += w0;                                    // the row of W's tensor map
      for (int kt = tile == first_tile ? ahead : 0; kt < k_tiles; ++kt) {
        if (round > 0 && !warp_wait(&empty_bar[s], (round & 1) ^ 1, status, T5_ERR_PRODUCER, abort_flag)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          expect(s);
          load_x(s, kt, m0);
          load_w(s, kt, n0);
        }
        __syncwarp();
        if (++s == stages) s = 0, ++round;
      }
    }
  } else if (warp == 1) {
    pdl_wait();
    pdl_trigger();
    // MMA issue: the whole warp runs the loop, one elected lane issues the instructions
    const uint32_t idesc = umma_idesc(T5_BM * CLUSTER, bn);
    const uint64_t desc0 = umma_desc_sw128(smem_u32(tiles));      // a step along the tiles adds (bytes >> 4)
    const int num_tiles = grouped ? groups.n_tiles[0] * tiles_n : num_tiles_plain;
    uint32_t local = 0;                            // tiles done by this block
    int s = 0, round = 0;
    bool ok = rank == 0;                           // (the second block of a pair issues nothing)
    for (int tile = first_tile; tile < num_tiles && ok; tile += tile_step, ++local) {
      const uint32_t buf = local & 1;
      // the epilogue must have drained this buffer (its previous use was tile local - 2)
      if (local >= 2 && !warp_wait(&acc_empty[buf], ((local >> 1) & 1) ^ 1, status, T5_ERR_MMA, abort_flag)) break;
      tcgen05_after_sync();
      const uint32_t acc = tmem_base + buf * 256;
      for (int kt = 0; kt < k_tiles; ++kt) {
        if (!warp_wait(&full_bar[s], round & 1, status, T5_ERR_MMA, abort_flag)) {
          ok = false;
          break;
        }
        tcgen05_after_sync();
        if (elect_one()) {
          const uint64_t a_desc = desc0 + ((static_cast<uint32_t>(s) * stage_bytes) >> 4);
          const uint64_t b_desc = a_desc + (T5_A_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < T5_BK / 16; ++k) {
            // 16 elements of K = 32 bytes further along the swizzled row
            if constexpr (PAIR) umma_bf16_pair(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);
            else umma_bf16(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);
          }
          if constexpr (PAIR) umma_commit_pair(&empty_bar[s]);      // arrives when these MMAs have read the stage
          else umma_commit(&empty_bar[s]);
        }
        __syncwarp();
        if (++s == stages) s = 0, ++round;
      }
      if (ok && elect_one()) {                     // arrives when every MMA issued so far has completed
        if constexpr (PAIR) umma_commit_pair(&acc_full[buf]);
        else umma_commit(&acc_full[buf]);
      }
      __syncwarp();
    }
  } else {
    pdl_wait();
    pdl_trigger();
    // epilogue: warp w may touch TMEM lanes 32 * (w % 4) .. + 31
    const int quarter = warp & 3;
    const int num_tiles = grouped ? groups.n_tiles[0] * tiles_n : num_tiles_plain;
    const int M_all = M;
    uint32_t local = 0;
    for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++local) {
      const uint32_t buf = local & 1;
      int m0, n0, w0, M;                           // M: one past the last row this tile may store
      coords(tile, num_tiles, &m0, &n0, &w0, &M);
      M = min(M, M_all);
      const int row = m0 + quarter * 32 + lane;
      if (!warp_wait(&acc_full[buf], (local >> 1) & 1, status, T5_ERR_EPILOGUE, abort_flag)) break;
      tcgen05_after_sync();
      const uint32_t lane_addr = tmem_base + buf * 256 + (static_cast<uint32_t>(quarter * 32) << 16);
      unsigned char* my_stage = store_stage + (warp - 2) * (T5_STORE_BYTES / 4);
      const int row0 = m0 + quarter * 32;
      const int n_end = min(swiglu ? gate_rows : N, n0 + n_per_tile);      // one past the last feature this tile may store
      if (swiglu && coeffs != nullptr) {
        // clamped halves with biases: a branch of its own, so that the plain epilogue stays as small as it was
        const float limit = coeffs[0], gate_scale = coeffs[1];
        const float* bias_g = coeffs + CLAMPED_HEADER;
        const float* bias_u = bias_g + gate_rows;            // (gate_rows is a multiple of 8)
        for (int c0 = 0; c0 < bn / 2 && row0 < M; c0 += 64) {
#pragma unroll 1
          for (int hh = 0; hh < 2; ++hh) {
            uint4 w[4];
            uint32_t g[32], u[32];
            tmem_ld32(lane_addr + c0 + hh * 32, g);
            tmem_ld32(lane_addr + bn / 2 + c0 + hh * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              const int f = n0 + c0 + hh * 32 + j;
              uint4 q = make_uint4(0u, 0u, 0u, 0u);
              if (f < gate_rows) {
                const float4 ga = *reinterpret_cast<const float4*>(bias_g + f), gb = *reinterpret_cast<const float4*>(bias_g + f + 4);
                const float4 ua = *reinterpret_cast<const float4*>(bias_u + f), ub = *reinterpret_cast<const float4*>(bias_u + f + 4);
                auto fin = [&](int e, float bg, float bu) {
                  return clamped_swiglu_bf16(__uint_as_float(g[j + e]) + bg, __uint_as_float(u[j + e]) + bu, limit, gate_scale);
                };
                q = make_uint4(pack2_bf16(fin(0, ga.x, ua.x), fin(1, ga.y, ua.y)), pack2_bf16(fin(2, ga.z, ua.z), fin(3, ga.w, ua.w)),
                               pack2_bf16(fin(4, gb.x, ub.x), fin(5, gb.y, ub.y)), pack2_bf16(fin(6, gb.z, ub.z), fin(7, gb.w, ub.w)));
              }
              w[j / 8] = q;
            }
            stage_half_row(w, my_stage, lane, hh);
          }
          store_staged_rows(my_stage, lane, static_cast<bf16*>(y), ldy, row0, M, n0 + c0, n_end);
        }
      } else if (swiglu) {
        bf16* out = static_cast<bf16*>(y);
        for (int c0 = 0; c0 < bn / 2 && row0 < M; c0 += 64) {
#pragma unroll 1
          for (int hh = 0; hh < 2; ++hh) {
            uint4 w[4];
            uint32_t g[32], u[32];
            tmem_ld32(lane_addr + c0 + hh * 32, g);
            tmem_ld32(lane_addr + bn / 2 + c0 + hh * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint32_t w4[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float g0 = __uint_as_float(g[j + 2 * e]), g1 = __uint_as_float(g[j + 2 * e + 1]);
                const float u0 = __uint_as_float(u[j + 2 * e]), u1 = __uint_as_float(u[j + 2 * e + 1]);
                w4[e] = pack2_bf16(__fdividef(g0, 1.0f + __expf(-g0)) * u0, __fdividef(g1, 1.0f + __expf(-g1)) * u1);
              }
              w[j / 8] = make_uint4(w4[0], w4[1], w4[2], w4[3]);
            }
            stage_half_row(w, my_stage, lane, hh);
          }
          store_staged_rows(my_stage, lane, out, ldy, row0, M, n0 + c0, n_end);   // a multiple of 8
        }
      } else if (mode == T5_OUT_QKV_ROPE) {
        // W = [Wq; Wk; Wv]: a tile holds whole heads (head_dim 64 or 128 divides the tile width). Thread = row:
        // the two members of rotary pair i of a head are columns i and i + head_dim / 2 of the same thread.
        const bool live = row < M;
        const int pos = live ? rope.positions[row] : 0;
        const size_t slot = live ? qkv_rope_slot(rope, row, pos) : 0;
        const float fpos = static_cast<float>(pos) * rope.pos_scale;
        const int hd = rope.head_dim;
        const float4* my_angles = rope.angles != nullptr && live
                                      ? reinterpret_cast<const float4*>(rope.angles + static_cast<size_t>(row) * (hd / 2))
                                      : nullptr;       // two (cos, sin) pairs per 16-byte load
        // A warp past the last row has nothing to read or write; a row past it inside a live warp is carried along
        // unrotated (its sines and cosines are not looked up or worked out).
        const bool warp_live = row - lane < M;
        for (int h0 = 0; warp_live && h0 < bn && n0 + h0 < N; h0 += hd) {
          const int head = (n0 + h0) / hd;                // q heads, then k heads, then v heads
          const bool rotated = head < rope.n_heads + rope.n_kv_heads;
          bf16* dst = nullptr;
          if (live) {
            if (head < rope.n_heads) {
              dst = static_cast<bf16*>(y) + static_cast<size_t>(row) * ldy + static_cast<size_t>(head) * hd;
            } else if (slot != QKV_NO_SLOT) {
              const bool is_k = head < rope.n_heads + rope.n_kv_heads;
              const int kvh = head - rope.n_heads - (is_k ? 0 : rope.n_kv_heads);
              dst = (is_k ? rope.k_cache : rope.v_cache) + (slot * rope.n_kv_heads + kvh) * hd;
            }
          }
          for (int piece = 0; piece < hd / 64; ++piece) {     // 32 pairs at a time
            uint32_t lo[32], hi[32];
            tmem_ld32(lane_addr + h0 + piece * 32, lo);
            tmem_ld32(lane_addr + h0 + hd / 2 + piece * 32, hi);
            tmem_ld_wait();
            // (cos, sin) of the piece's 32 pairs, two pairs per float4: all requested before any is used
            float4 cs[16];
            if (rotated && live) {
              if (my_angles != nullptr) {
#pragma unroll
                for (int i = 0; i < 16; ++i) cs[i] = my_angles[piece * 16 + i];
              } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  sincosf(fpos * rope.inv_freq[piece * 32 + 2 * i], &cs[i].y, &cs[i].x);
                  sincosf(fpos * rope.inv_freq[piece * 32 + 2 * i + 1], &cs[i].w, &cs[i].z);
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) cs[i] = make_float4(1.0f, 0.0f, 1.0f, 0.0f);     // v heads: no rotation
            }
            uint4 wlo[4], whi[4];
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint32_t pl[4], ph[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float a0 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(lo[j + 2 * e])));
                const float a1 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(lo[j + 2 * e + 1])));
                const float b0 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(hi[j + 2 * e])));
                const float b1 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(hi[j + 2 * e + 1])));
                const float4 t4 = cs[j / 2 + e];
                pl[e] = pack2_bf16(a0 * t4.x - b0 * t4.y, a1 * t4.z - b1 * t4.w);
                ph[e] = pack2_bf16(a0 * t4.y + b0 * t4.x, a1 * t4.w + b1 * t4.z);
              }
              wlo[j / 8] = make_uint4(pl[0], pl[1], pl[2], pl[3]);
              whi[j / 8] = make_uint4(ph[0], ph[1], ph[2], ph[3]);
            }
            store_rows_pieces(wlo, whi, my_stage, lane, dst, piece * 32, hd / 2 + piece * 32);
          }
        }
      } else if (mode == T5_OUT_PAIRS) {
        // rows 2j and 2j + 1 of W are the gate and up rows of feature j: 128 columns of the tile give 64 of the output
        for (int c0 = 0; c0 < bn && row0 < M; c0 += 128) {
#pragma unroll 1
          for (int hh = 0; hh < 2; ++hh) {
            uint4 w[4];
            uint32_t v[2][32];
            tmem_ld32(lane_addr + c0 + hh * 64, v[0]);
            tmem_ld32(lane_addr + c0 + hh * 64 + 32, v[1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              auto fin = [&](int j) {
                const float g = __uint_as_float(v[i / 2][i % 2 * 16 + j]);
                return __fdividef(g, 1.0f + __expf(-g)) * __uint_as_float(v[i / 2][i % 2 * 16 + j + 1]);
              };
              w[i] = make_uint4(pack2_bf16(fin(0), fin(2)), pack2_bf16(fin(4), fin(6)), pack2_bf16(fin(8), fin(10)), pack2_bf16(fin(12), fin(14)));
            }
            stage_half_row(w, my_stage, lane, hh);
          }
          store_staged_rows(my_stage, lane, static_cast<bf16*>(y), ldy, row0, M, (n0 + c0) / 2, N / 2);   // N / 2 is a multiple of 8
        }
      } else if (mode == T5_OUT_F32) {
        for (int c0 = 0; c0 < bn && row0 < M; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(lane_addr + c0, v);
          tmem_ld_wait();
          if (row >= M) continue;
          float* out = static_cast<float*>(y) + static_cast<size_t>(row) * ldy;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const int col = n0 + c0 + j;
            if (col < n_end) {                     // a multiple of 4 in this mode
              const float4 add = coeffs != nullptr ? *reinterpret_cast<const float4*>(coeffs + col) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
              *reinterpret_cast<float4*>(out + col) =
                  make_float4(fmaf(__uint_as_float(v[j]), out_scale, add.x), fmaf(__uint_as_float(v[j + 1]), out_scale, add.y),
                              fmaf(__uint_as_float(v[j + 2]), out_scale, add.z), fmaf(__uint_as_float(v[j + 3]), out_scale, add.w));
            }
          }
        }
      } else {
        // bf16 out, or on the way the squared ReLU of an ungated feed-forward, its GELU in the tanh form or xIELU (whose two
        // coefficients lie in memory). Every one a loop of its own, 32 columns long: with the activations' code between the plain
        // store's instructions (skipped, number by number) a tile's epilogue was bound by fetching instructions (1777 x 2048 x 2048, in a row: 20.1 us a product, now 15.1).
        auto write = [&](auto fin) {
          for (int c0 = 0; c0 < bn && row0 < M; c0 += 64) {
#pragma unroll 1
            for (int hh = 0; hh < 2; ++hh) {
              uint4 w[4];
              uint32_t v[32];
              tmem_ld32(lane_addr + c0 + hh * 32, v);
              tmem_ld_wait();
              auto two = [&](int j) { return pack2_bf16(fin(__uint_as_float(v[j])), fin(__uint_as_float(v[j + 1]))); };
#pragma unroll
              for (int j = 0; j < 32; j += 8) w[j / 8] = make_uint4(two(j), two(j + 2), two(j + 4), two(j + 6));
              stage_half_row(w, my_stage, lane, hh);
            }
            store_staged_rows(my_stage, lane, static_cast<bf16*>(y), ldy, row0, M, n0 + c0, n_end);   // a multiple of 8
          }
        };
        if (mode == T5_OUT_RELU2) {
          write([&](float v) { v = fmaxf(v * out_scale, 0.0f); return v * v; });
        } else if (mode == T5_OUT_GELU) {
          write([&](float v) { return gelu_tanh_bf16(v * out_scale); });
        } else if (mode == T5_OUT_XIELU) {
          const float c0_x = coeffs[0], c1_x = coeffs[1];
          write([&](float v) { return xielu_bf16(v, c0_x, c1_x); });
        } else {
          write([&](float v) { return v * out_scale; });
        }
      }
      // this warp has read its part of the buffer: let the MMA warp reuse it
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_first_block(&acc_empty[buf]);
        else mbar_arrive(&acc_empty[buf]);
      }
    }
  }
  // common exit: every role arrives here, with or without a timeout
  drain_after_abort(abort_flag);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();              // nobody leaves while its partner may still send to it or read from it
  if (warp == 1) {
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(T5_TMEM_COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(T5_TMEM_COLS) : "memory");
  }
}

// ---- host side -------------------------------------------------------------------------------------

// rows x cols bf16, row pitch `ld` elements, box = box_rows x 64 columns, 128-byte swizzle, zero fill outside.
static inline int make_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (fn == nullptr) return DL_ERR_UNSUPPORTED;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(T5_BK), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 700000 + static_cast<int>(r);
}

}  // namespace dl

// What a slice of 64 k takes a round of tiles of bn columns, of blocks alone or of pairs, in us: from products of 543 to 2,048
// rows by 2,048 or 3,072 features, between K 2048 and K 8192, on B200. At 35 products from 64 to 2,048 rows the width and kind
// with the least rounds x cost is the fastest measured or within 5 % of it. Against blocks alone at 256, 192 or 128 columns,
// with pairs that only shared W's loads for the largest products (us, cold caches, same order of sums): 2048 x 16384 (SwiGLU) x
// 2048 98 -> 86; 2048 x 2048 x 8192 70 -> 57; 2499 x 28672 (SwiGLU) x 4096 395 -> 382; 2499 x 4096 x 14336 230 -> 202. (K in 2
// to 8 pieces over a cluster, the sums added through distributed shared memory, takes 25.5 us for 700 x 2048 x 8192 against
// 29.8 here, but no whole step gained from it by more than its runs differ.)
static double t5_slice_us(int bn, bool pair) {
  static const double alone[] = {0.215, 0.222, 0.244, 0.293, 0.321, 0.361, 0.402};       // 64, 96, .. 256
  static const double paired[] = {0.183, 0.190, 0.209, 0.240, 0.268, 0.295, 0.325};
  return (pair ? paired : alone)[(bn - 64) / 32];
}

struct T5Choice {
  int bn;
  bool pair;
};

// The width and kind of tile whose rounds over the SMs cost least. SwiGLU pairs gate and up columns, so a tile holds bn / 2
// features; the q | k | v epilogue needs whole heads (or, at head size 128, whole tiles of heads) in a tile.
// pairs: 0 never, 1 always, -1 by cost.
static T5Choice t5_choose(long long m_blocks, int feats, int mode, int head_dim, int sms, int pairs) {
  // DYNALM_GEMM_TILE=<multiple of 32, 64 to 256> overrides the width where it is allowed
  static int forced = -1;
  if (forced < 0) {
    const char* e = getenv("DYNALM_GEMM_TILE");
    forced = e ? atoi(e) : 0;
  }
  T5Choice best = {256, false};
  double least = 1e300;
  for (int pair = 0; pair < 2; ++pair) {
    if (pairs >= 0 && pairs != pair) continue;
    for (int bn = 256; bn >= 64; bn -= 32) {
      if (mode == dl::T5_OUT_QKV_ROPE && bn % head_dim != 0) continue;
      if (forced >= 64 && forced <= 256 && forced % 32 == 0 && forced != bn && (mode != dl::T5_OUT_QKV_ROPE || forced % head_dim == 0)) continue;
      const int per = mode == dl::T5_OUT_SWIGLU ? bn / 2 : bn;
      const long long t = (m_blocks + pair) / (1 + pair) * ((feats + per - 1) / per);
      const int units = sms / (1 + pair);
      const double c = static_cast<double>((t + units - 1) / units) * t5_slice_us(bn, pair != 0);
      if (c < least) {
        least = c;
        best = {bn, pair != 0};
      }
    }
  }
  return best;
}

template <bool PAIR>
static int t5_run(cudaLaunchConfig_t cfg, const CUtensorMap& map_x, const CUtensorMap& map_w, void* y, int ldy, int M, int N,
                  int K, int mode, float out_scale, int gate_rows, int tiles_n, int tiles, int group_m, int* status,
                  const dl::QkvRope& rope, const dl::T5Groups& groups, const float* coeffs, int bn) {
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(dl::gemm_tcgen05_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(dl::T5_SMEM));
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  cfg.dynamicSmemBytes = dl::T5_SMEM;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, dl::gemm_tcgen05_kernel<PAIR>, map_x, map_w, y, ldy, M, N, K, mode, out_scale,
                                             gate_rows, tiles_n, tiles, group_m, status, rope, groups, coeffs, bn));
}

// x: bf16 [M, K] rows of ldx elements; w: bf16 [N, K] contiguous; both 16-byte aligned with K and ldx multiples of 8.
// mode 0: y bf16 [M, N] (N % 8 == 0); mode 1: y fp32 [M, N] (N % 4 == 0); mode 2: w = [gate; up] with N = 2F rows,
// y bf16 [M, F] = silu(x Wg^T) * (x Wu^T) (F % 8 == 0), or with coeffs (N + 4 float32, 16-byte aligned: common.cuh,
// CLAMPED_HEADER) the gated activation with clamped halves and biases; mode 4: y bf16 [M, N] = max(x W^T, 0)^2; mode 5: = gelu_tanh(x W^T);
// mode 7: = xIELU(x W^T) with coeffs = two float32 on the device; mode 1 with coeffs: N float32 (16-byte aligned) that are added. status: one device int, set to a nonzero code if a wait
// inside the kernel timed out (left untouched otherwise).
static int t5_launch(const void* x, int ldx, const void* w, void* y, int ldy, int M, int N, int K, int mode, float out_scale,
                     int* status, const dl::QkvRope& rope, int pairs, cudaStream_t stream, const float* coeffs = nullptr) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (K & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) ||
      status == nullptr || mode < 0 || (mode > 5 && mode != dl::T5_OUT_XIELU) || (mode == dl::T5_OUT_XIELU && coeffs == nullptr))
    return DL_ERR_UNSUPPORTED;
  if ((mode == dl::T5_OUT_SWIGLU || mode == dl::T5_OUT_F32) && (reinterpret_cast<uintptr_t>(coeffs) & 15)) return DL_ERR_UNSUPPORTED;
  const int feats = mode == dl::T5_OUT_SWIGLU ? N / 2 : N;
  if ((mode == dl::T5_OUT_SWIGLU && (N & 1)) || (mode == dl::T5_OUT_F32 ? (feats & 3) || (ldy & 3) : (feats & 7) || (ldy & 7)) ||
      (reinterpret_cast<uintptr_t>(y) & 15))
    return DL_ERR_UNSUPPORTED;
  const int sms = dl::sm_count();
  const long long m_blocks = (M + dl::T5_BM - 1) / dl::T5_BM;
  const T5Choice choice = t5_choose(m_blocks, feats, mode, rope.head_dim, sms, pairs);
  const int cluster = choice.pair ? 2 : 1, bn = choice.bn;
  const long long m_tiles = (m_blocks + cluster - 1) / cluster;
  const int units = sms / cluster;                                          // blocks, or pairs of them
  const int per_tile = mode == dl::T5_OUT_SWIGLU ? bn / 2 : bn;
  const int tiles_n = (feats + per_tile - 1) / per_tile;
  const long long tiles = m_tiles * tiles_n;
  if (tiles > (1ll << 30)) return DL_ERR_UNSUPPORTED;
  CUtensorMap map_x, map_w;
  int rc = dl::make_map(&map_x, x, M, K, ldx, dl::T5_BM);
  if (rc != 0) return rc;
  rc = dl::make_map(&map_w, w, N, K, K, bn / 2);
  if (rc != 0) return rc;
  // Row blocks to a group of tiles (t5_tile_coords): as many as keep the group's rows of x within about 32 MB of L2,
  // 4 to 16. DYNALM_GEMM_GROUP_M overrides it (1: along the columns first).
  static int forced_group = -1;
  if (forced_group < 0) { const char* e = getenv("DYNALM_GEMM_GROUP_M"); forced_group = e ? atoi(e) : 0; }
  long long group = (32ll << 20) / (2ll * dl::T5_BM * cluster * K);
  group = group < 4 ? 4 : (group > 16 ? 16 : group);
  if (forced_group > 0) group = forced_group;
  const int group_m = static_cast<int>(group < m_tiles ? group : m_tiles);
  const int blocks = static_cast<int>(tiles < units ? tiles : units) * cluster;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(dl::T5_THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (choice.pair) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 2;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (dl::pdl_mode() >= 1) {      // the kernel may start before the one in front has ended: it requests W before its wait
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  const int gate_rows = mode == dl::T5_OUT_SWIGLU ? N / 2 : 0;
  const dl::T5Groups plain = {nullptr, nullptr, 0};
  return choice.pair ? t5_run<true>(cfg, map_x, map_w, y, ldy, M, N, K, mode, out_scale, gate_rows, tiles_n, static_cast<int>(tiles),
                                    group_m, status, rope, plain, coeffs, bn)
                     : t5_run<false>(cfg, map_x, map_w, y, ldy, M, N, K, mode, out_scale, gate_rows, tiles_n, static_cast<int>(tiles),
                                     group_m, status, rope, plain, coeffs, bn);
}

// A grouped product (see T5Groups): a bf16 [rows, K] whose runs of rows are listed in `tiles`, w bf16 [matrices, N, K]
// contiguous, y [rows, N] bf16 (mode 0, or 4 with the squared ReLU) or fp32 (mode 1), or with mode 6 (gate and up rows of w
// in turn, N a multiple of 16) y [rows, N / 2] bf16. max_row_tiles: the most row tiles
// the list can hold; the grid is sized for it and blocks past the list's end do nothing.
static int t5_launch_grouped(const void* a, int lda, int rows, const void* w, int matrices, int N, int K, void* y, int ldy,
                             int mode, const int* tiles, const int* n_tiles, int max_row_tiles, int* status,
                             cudaStream_t stream) {
  if (rows <= 0 || N <= 0 || max_row_tiles <= 0) return 0;
  if (K <= 0 || (K & 7) || (lda & 7) || (reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(w) & 15) ||
      (reinterpret_cast<uintptr_t>(y) & 15) || status == nullptr || tiles == nullptr || n_tiles == nullptr || matrices <= 0 ||
      (mode != dl::T5_OUT_BF16 && mode != dl::T5_OUT_F32 && mode != dl::T5_OUT_RELU2 && mode != dl::T5_OUT_PAIRS) ||
      (mode == dl::T5_OUT_PAIRS && (N & 15)) ||
      (mode == dl::T5_OUT_F32 ? (N & 3) || (ldy & 3) : (N & 7) || (ldy & 7)) ||
      static_cast<long long>(matrices) * N > (1ll << 30))
    return DL_ERR_UNSUPPORTED;
  const int bn = N >= 256 ? 256 : 128;
  const int tiles_n = (N + bn - 1) / bn;
  const long long most = static_cast<long long>(max_row_tiles) * tiles_n;
  if (most > (1ll << 30)) return DL_ERR_UNSUPPORTED;
  CUtensorMap map_x, map_w;
  int rc = dl::make_map(&map_x, a, rows, K, lda, dl::T5_BM);
  if (rc != 0) return rc;
  rc = dl::make_map(&map_w, w, matrices * N, K, K, bn / 2);
  if (rc != 0) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(most < dl::sm_count() ? most : dl::sm_count()));
  cfg.blockDim = dim3(dl::T5_THREADS);
  cfg.stream = stream;
  const dl::QkvRope none = {};
  const dl::T5Groups groups = {tiles, n_tiles, N};
  return t5_run<false>(cfg, map_x, map_w, y, ldy, rows, N, K, mode, 1.0f, 0, tiles_n, 0, 1, status, none, groups, nullptr, bn);
}

// Fills the epilogue's parameters for the q | k | v product and launches it (see dl_gemm_tcgen05_qkv_rope).
static int t5_launch_qkv_rope(const void* x, int ldx, const void* w, void* q_out, int ldq, int M, int K, const int* positions,
                              const int* row_request, const int* block_table, int max_blocks, void* k_cache, void* v_cache,
                              const float* inv_freq, const void* angles, float pos_scale, int n_heads, int n_kv_heads,
                              int head_dim, int page_size, int* status, int pairs, cudaStream_t stream) {
  if ((head_dim != 64 && head_dim != 128) || n_heads <= 0 || n_kv_heads <= 0 || page_size <= 0 || inv_freq == nullptr ||
      (reinterpret_cast<uintptr_t>(k_cache) & 15) || (reinterpret_cast<uintptr_t>(v_cache) & 15) ||
      (reinterpret_cast<uintptr_t>(angles) & 15))
    return DL_ERR_UNSUPPORTED;
  dl::QkvRope p;
  p.positions = positions;
  p.row_request = row_request;
  p.block_table = block_table;
  p.max_blocks = max_blocks;
  p.k_cache = static_cast<dl::bf16*>(k_cache);
  p.v_cache = static_cast<dl::bf16*>(v_cache);
  p.inv_freq = inv_freq;
  p.angles = static_cast<const float2*>(angles);
  p.pos_scale = pos_scale;
  p.n_heads = n_heads;
  p.n_kv_heads = n_kv_heads;
  p.head_dim = head_dim;
  p.page_size = page_size;
  return t5_launch(x, ldx, w, q_out, ldq, M, (n_heads + 2 * n_kv_heads) * head_dim, K, dl::T5_OUT_QKV_ROPE, 1.0f, status, p,
                   pairs, stream);
}
