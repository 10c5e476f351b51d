// int4 x int4 GEMM with the dequantising epilogue on pairs of CTAs (tcgen05 cta_group::2), A as int8 in operand order.
// Included by gemm_i4.cu inside namespace qb, before the host side.
//
// A cluster of two CTAs (two SMs) owns a tile of 256 rows x up to 256 columns.  Each CTA copies its 128 A rows (int8, by
// TMA straight into the operand ring) and copies and unpacks HALF of the tile's B rows; one MMA (M 256, N up to 256, K 32)
// reads both CTAs' shared memory and leaves 128 rows of the result in each CTA's tensor memory.
//
// Why pairs: the 256 x 256 tile of one CTA (gemm_i4_wide_kernel) needs all 512 tensor-memory columns, so its epilogue is
// exposed after every tile, and every CTA unpacks all 256 B rows.  Here an SM holds 256 columns per tile: two accumulator
// buffers fit and the epilogue of a tile runs behind the MMAs of the next, while the B traffic per MAC (packed read, int8
// write, MMA read) through each SM's shared memory is halved.
//
// What bounds it: the issue of the MMAs, then the power limit.  Four MMAs of 256 columns need 512 cycles of the tensor
// pipe; issued from a `lane == 0` branch a 128-K step took 1250 cycles with .release.cluster arrivals, 700 with plain ones,
// and takes 260 + 1.3 per column with the warp-uniform loop below.  Measured (GEMM alone, launches back to back, all operands
// from HBM), the one-CTA 256 x 256 kernel on the same int8 operand against this one: K 4096, M 2048 N 4096 28.3 -> 26.3 us
// (2609 TOPS), N 11008 74.0 -> 54.8, N 12288 78.9 -> 62.2; M 8192 N 4096 103 -> 79.5, N 12288 300 -> 225 (3670 TOPS).
#pragma once

namespace pair2 {
constexpr int TM = 256, TN = 256;              // tile of the pair
constexpr int CTA_ROWS = TM / 2;               // A rows, and rows of the result, per CTA
constexpr int MAX_B_ROWS = TN / 2;             // B rows a CTA copies and unpacks
constexpr int STAGES = 5;                      // operand ring: 16 KB A + 16 KB B (int8) per stage
constexpr int P_STAGES = 5;                    // packed B ring: 8 KB per stage
constexpr int A_BYTES = CTA_ROWS * U8_ROW;
constexpr int B_BYTES = MAX_B_ROWS * U8_ROW;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int P_BYTES = MAX_B_ROWS * PK_ROW;
constexpr int kEpiWarps = 8, kFirstEpi = 2;
constexpr int kUnpackWarps = 8, kFirstUnpack = kFirstEpi + kEpiWarps;
constexpr int kUnpackGroup = 4;                // warps that unpack one stage; the two groups take turns
constexpr int kAWarp = kFirstUnpack + kUnpackWarps;
constexpr int kWarps = kAWarp + 1;
constexpr int kThreads = kWarps * 32;
constexpr int SLAB_BYTES = 32 * 64;            // one output piece: 32 rows x 32 columns of bf16
constexpr int SLABS_BYTES = kEpiWarps * SLAB_BYTES;
constexpr int VEC_STRIDE = TN * 12;            // per accumulator buffer: b_add (int32), b_mul and bias (fp32) of the tile
constexpr int NUM_BARS = 2 * P_STAGES + 2 * STAGES + 4 + 1;
constexpr int LAYOUT_BYTES = STAGES * STAGE_BYTES + P_STAGES * P_BYTES + SLABS_BYTES + 2 * VEC_STRIDE + NUM_BARS * 8 + 16;
constexpr int SMEM_BYTES = LAYOUT_BYTES + 1024;
static_assert(SMEM_BYTES <= 232448, "layout does not fit");
static_assert(STAGES * STAGE_BYTES >= kEpiWarps * 4 * SLAB_BYTES, "the last tile's pieces are staged in the operand ring");
constexpr uint32_t IDESC_BASE = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TM >> 4) << 24);  // + (width >> 3) << 17
// Tile number -> tile row and column range.  The tiles are walked in groups of `group` tile rows, all columns of a group
// before the next, rows first: the tiles in flight share few A rows and few weight columns.  Tile columns are multiples
// of 32 wide (the N granularity of this MMA, and whole 32-column output pieces).
__device__ __forceinline__ void tile_at(const EpilogueParams& ep, int tile, int tiles_m, int group, int& mt, int& n0, int& bn) {
    const int g = tile / (group * ep.col_count);
    const int rows = min(group, tiles_m - g * group);
    const int in_group = tile - g * group * ep.col_count;
    const int col = in_group / rows;
    mt = g * group + in_group - col * rows;
    const int wider = col < ep.col_rem ? col : ep.col_rem;
    n0 = (col * ep.col_units + wider) << 5;
    bn = (ep.col_units + (col < ep.col_rem ? 1 : 0)) << 5;
}
}  // namespace pair2

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair2::kThreads, 1)
gemm_i4_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_d, const __grid_constant__ EpilogueParams ep, const int M,
                    const int N, const int K, const int b_box_rows, const int group) {
    using namespace pair2;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_base = smem_u32(smem_raw);
    const uint32_t smem_base = (raw_base + 1023u) & ~1023u;  // the same offset in both CTAs (the MMA relies on it)
    const uint32_t p_base = smem_base + STAGES * STAGE_BYTES;
    const uint32_t slab_base = p_base + P_STAGES * P_BYTES;
    const uint32_t vec_base = slab_base + SLABS_BYTES;
    const uint32_t full_p = vec_base + 2 * VEC_STRIDE;   // packed piece has landed (this CTA)
    const uint32_t empty_p = full_p + 8 * P_STAGES;      // packed piece has been unpacked (this CTA)
    const uint32_t full = empty_p + 8 * P_STAGES;        // even CTA: A of both CTAs has landed, B of both is unpacked
    const uint32_t empty = full + 8 * STAGES;            // both CTAs: the MMAs have read the stage
    const uint32_t tmem_full = empty + 8 * STAGES;       // both CTAs: accumulator buffer complete
    const uint32_t tmem_empty = tmem_full + 16;          // even CTA: both CTAs' epilogues have read the buffer
    const uint32_t mma_done = tmem_empty + 16;
    const uint32_t tmem_slot = mma_done + 8;
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - raw_base));
    volatile int* epi_abort = reinterpret_cast<volatile int*>(smem_raw + (tmem_slot + 8 - raw_base));  // see gemm_i4_kernel

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // uniform, and known to be
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int tiles_m = (M + TM - 1) / TM;
    const int num_tiles = tiles_m * ep.col_count;
    const int num_kb = (K + BK - 1) / BK;
    const uint32_t p_bytes = (uint32_t)b_box_rows * PK_ROW;
    uint32_t pre_issued = 0;

    if (threadIdx.x == 0) {
        QB_TRACE(0);
        for (int i = 0; i < P_STAGES; ++i) {
            mbar_init(full_p + 8 * i, 1);
            mbar_init(empty_p + 8 * i, kUnpackGroup);
        }
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(full + 8 * i, 1 + 2 * kUnpackGroup);
            mbar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(tmem_full + 8 * i, 1);
            mbar_init(tmem_empty + 8 * i, 2 * kEpiWarps);
        }
        mbar_init(mma_done, 1);
        fence_barrier_init();
        *epi_abort = 0;
        // The first weight copies leave before tensor memory is allocated and the CTAs have met.
        if (pair < num_tiles) {
            tma_prefetch_desc(&tmap_b);
            int mt, n0, bn;
            tile_at(ep, pair, tiles_m, group, mt, n0, bn);
            for (; pre_issued < (uint32_t)P_STAGES && (int)pre_issued < num_kb; ++pre_issued) {
                mbar_arrive_expect_tx(full_p + 8 * pre_issued, p_bytes);
                tma_load_2d(p_base + pre_issued * P_BYTES, &tmap_b, (int)pre_issued * PK_ROW, n0 + (int)rank * (bn >> 1), full_p + 8 * pre_issued);
            }
        }
    }
    __syncwarp();
    cluster_sync();  // both CTAs have started and initialised their barriers: an allocation for the pair involves the other CTA
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // tensor memory is allocated in both
    tc_fence_after();
    const uint32_t tmem_acc = *tmem_slot_ptr;
    let_dependents_launch();  // only now that tensor memory is allocated (see gemm_i4_kernel)

    if (warp == 0) {
        // ------------------------------ packed B producer (each CTA its half of the tile's B rows) ------------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
                int mt, n0, bn;
                tile_at(ep, tile, tiles_m, group, mt, n0, bn);
                const int b_row = n0 + (int)rank * (bn >> 1);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    if (it < pre_issued) continue;
                    const uint32_t s = it % P_STAGES, ph = (it / P_STAGES) & 1u;
                    if (!(ok = mbar_wait(empty_p + 8 * s, ph ^ 1u, 31))) break;
                    mbar_arrive_expect_tx(full_p + 8 * s, p_bytes);
                    tma_load_2d(p_base + s * P_BYTES, &tmap_b, kb * PK_ROW, b_row, full_p + 8 * s);
                }
            }
            const uint32_t pending = it < (uint32_t)P_STAGES ? it : (uint32_t)P_STAGES;
            for (uint32_t j = 0; j < pending; ++j) {  // do not leave while a copy of ours may still land
                const uint32_t i2 = it - 1 - j;
                mbar_wait(full_p + 8 * (i2 % P_STAGES), (i2 / P_STAGES) & 1u, 32);
            }
        }
    } else if (warp == kAWarp) {
        // ------------------------------ A producer (each CTA its 128 rows; the even CTA's barrier counts both) ------
        if (lane == 0) {
            tma_prefetch_desc(&tmap_a);
            wait_for_preceding_grid();  // the A operand is the quantiser's output
            uint32_t it = 0;
            bool ok = true;
            for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
                int mt, n0, bn;
                tile_at(ep, tile, tiles_m, group, mt, n0, bn);
                const int m0 = mt * TM + (int)rank * CTA_ROWS;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const uint32_t s = it % STAGES, ph = (it / STAGES) & 1u;
                    if (!(ok = mbar_wait(empty + 8 * s, ph ^ 1u, 33))) break;
                    if (rank == 0) mbar_arrive_expect_tx(full + 8 * s, 2 * A_BYTES);
                    tma_load_2d_pair(smem_base + s * STAGE_BYTES, &tmap_a, kb * U8_ROW, m0, map_to_cta(full + 8 * s, 0));
                }
            }
            if (ok) {
                // Every stage has been read, so every copy has landed and no MMA arrives on this CTA's barriers any more.
                const uint32_t pending = it < (uint32_t)STAGES ? it : (uint32_t)STAGES;
                for (uint32_t j = 0; j < pending; ++j) {
                    const uint32_t i2 = it - 1 - j;
                    mbar_wait(empty + 8 * (i2 % STAGES), (i2 / STAGES) & 1u, 40);
                }
            } else {  // a bounded wait gave up: give copies in flight (microseconds) a millisecond to land
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer (even CTA; all lanes walk the loop, see elect_one) --------------
        if (rank == 0) {
            const uint64_t desc0 = make_smem_desc(smem_base);
            uint32_t s = 0, ph = 0, local_tile = 0;
            bool ok = true;
            for (int tile = pair; tile < num_tiles && ok; tile += pairs, ++local_tile) {
                const uint32_t acc = local_tile & 1u, acc_ph = (local_tile >> 1) & 1u;
                int mt, n0, bn;
                tile_at(ep, tile, tiles_m, group, mt, n0, bn);
                const uint32_t idesc = IDESC_BASE | ((uint32_t)(bn >> 3) << 17);
                ok = __all_sync(0xffffffffu, mbar_wait(tmem_empty + 8 * acc, acc_ph ^ 1u, 34));
                tc_fence_after();
                const uint32_t d_tmem = tmem_acc + acc * TN;
                for (int kb = 0; kb < num_kb && ok; ++kb) {
                    ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, ph, 35));
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t da = desc0 + (uint64_t)(s * (STAGE_BYTES >> 4)), db = da + (A_BYTES >> 4);
                    if (elect_one()) {
                        umma_i8_pair(d_tmem, da, db, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
                        for (int j = 1; j < BK / 32; ++j) umma_i8_pair(d_tmem, da + 2 * j, db + 2 * j, idesc, 1u);
                        umma_commit_pair(empty + 8 * s);
                    }
                    __syncwarp();
                    if (++s == STAGES) s = 0, ph ^= 1u;
                }
                if (ok && elect_one()) umma_commit_pair(tmem_full + 8 * acc);
                __syncwarp();
            }
            if (elect_one()) umma_commit_pair_local(mma_done);
            __syncwarp();
            mbar_wait(mma_done, 0, 36);
            QB_TRACE(2);
        }
    } else if (warp < kFirstUnpack) {
        // ------------------------------ epilogue ------------------------------
        const int quad = warp & 3;                    // tensor-memory lane quadrant this warp may read
        const int half = (warp - kFirstEpi) >> 2;     // which half of the tile's 32-column pieces
        const int et = threadIdx.x - kFirstEpi * 32;  // 0 .. 255
        const uint32_t own_slab = slab_base + (uint32_t)(warp - kFirstEpi) * SLAB_BYTES;
        const uint32_t ring_slab = smem_base + (uint32_t)(warp - kFirstEpi) * (4 * SLAB_BYTES);
        const uint32_t slab_row = (uint32_t)lane * 64u, slab_xor = ((uint32_t)lane >> 1) & 3u;  // 64-byte swizzle
        const uint32_t leader_empty = map_to_cta(tmem_empty, 0);
        uint32_t local_tile = 0;
        wait_for_preceding_grid();  // the row sums and scales come from the quantiser
        for (int tile = pair; tile < num_tiles; tile += pairs, ++local_tile) {
            const uint32_t acc = local_tile & 1u, acc_ph = (local_tile >> 1) & 1u;
            int mt, n0, bn;
            tile_at(ep, tile, tiles_m, group, mt, n0, bn);
            const int warp_row0 = mt * TM + (int)rank * CTA_ROWS + quad * 32;
            const int row = warp_row0 + lane;
            const bool row_ok = row < M;
            int* sb_add = reinterpret_cast<int*>(smem_raw + (vec_base - raw_base) + acc * VEC_STRIDE);
            float* sb_mul = reinterpret_cast<float*>(sb_add + TN);
            float* sb_bias = sb_mul + TN;
            {
                const bool in = et < bn && n0 + et < N;
                sb_add[et] = in ? ep.b_add[n0 + et] : 0;
                sb_mul[et] = in ? bf16_to_f32(ep.b_mul[n0 + et]) : 0.f;
                if (ep.bias != nullptr) sb_bias[et] = in ? bf16_to_f32(ep.bias[n0 + et]) : 0.f;
            }
            int a_add = 0;
            float half_a_mul = 0.f;
            if (row_ok) {
                a_add = ep.a_add[row];
                half_a_mul = 0.5f * bf16_to_f32(ep.a_mul[row]);
            }
            if (!mbar_wait(tmem_full + 8 * acc, acc_ph, 37)) *epi_abort = 1;
            // vectors staged (a buffer is rewritten two tiles later, behind this barrier of the tile between); uniform give-up
            asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
            if (*epi_abort) break;
            tc_fence_after();
            const uint32_t t_row = tmem_acc + ((uint32_t)(quad * 32) << 16) + acc * TN;
            const bool last = tile + pairs >= num_tiles;  // the operand ring is idle: every piece has a slab of its own there
            const int pieces = bn >> 5, first = half == 0 ? 0 : (pieces + 1) >> 1, end = half == 0 ? (pieces + 1) >> 1 : pieces;
#pragma unroll 1
            for (int pc = first; pc < end; ++pc) {
                const int c0 = pc * 32;
                if (n0 + c0 >= N || warp_row0 >= M) break;  // warp-uniform
                uint32_t r[32];
                tmem_ld32(t_row + c0, r);
                tmem_ld_wait32(r);
                uint32_t w[16];
                dequant_chunk(r, a_add, half_a_mul, sb_add + c0, sb_mul + c0, w);
                if (ep.bias != nullptr) add_bias_chunk(w, sb_bias + c0);
                if (!ep.tma_store) {
                    if (row_ok) store_bf16_chunk(w, ep, row, n0 + c0, N);
                    continue;
                }
                const uint32_t slab = last ? ring_slab + (uint32_t)(pc - first) * SLAB_BYTES : own_slab;
                if (!last) {
                    if (lane == 0) bulk_wait_read_all();  // the previous piece has left the slab
                    __syncwarp();
                }
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    sts128(slab + slab_row + ((j ^ slab_xor) << 4), make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]));
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(&tmap_d, slab, n0 + c0, warp_row0);
                    bulk_commit_group();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_empty + 8 * acc);
            if (warp == kFirstEpi && lane == 0) QB_TRACE(3);
        }
        if (lane == 0) bulk_wait_read_all();  // the slabs have been read before the CTA ends
    } else {
        // ------------------------------ unpack warps ------------------------------
        const int grp = (warp - kFirstUnpack) / kUnpackGroup;  // takes every second stage
        const int t = (threadIdx.x - kFirstUnpack * 32) & (kUnpackGroup * 32 - 1);  // 0 .. 127
        uint32_t it = 0;
        bool ok = true;
        for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
            int mt, n0, bn;
            tile_at(ep, tile, tiles_m, group, mt, n0, bn);
            const int b_rows = bn >> 1;  // a multiple of 16: the row test below is warp-uniform
            for (int kb = 0; kb < num_kb; ++kb, ++it) {
                if ((int)(it & 1u) != grp) continue;
                const uint32_t ps = it % P_STAGES, pph = (it / P_STAGES) & 1u;
                const uint32_t us = it % STAGES, uph = (it / STAGES) & 1u;
                // The operand stage first: the MMAs of step it - STAGES have then completed, so every copy up to that step has
                // landed, slot ps is in the phase this step waits for, and its parity names only that one.  The other way
                // round nothing has ended the slot's use before, which was the OTHER group's (P_STAGES is odd): a late copy
                // leaves the barrier a phase behind, whose parity is the same, and the wait returns at once.
                static_assert(STAGES <= P_STAGES, "a packed slot's use before this one has ended");
                ok = mbar_wait(empty + 8 * us, uph ^ 1u, 39) && mbar_wait(full_p + 8 * ps, pph, 38);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const uint32_t src = p_base + ps * P_BYTES;
                const uint32_t dst = smem_base + us * STAGE_BYTES + A_BYTES;
                constexpr int ITEMS = MAX_B_ROWS * 4 / (kUnpackGroup * 32);  // 4 pieces of 16 packed bytes per thread
                uint4 pk[ITEMS];
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    const int item = t + i * kUnpackGroup * 32;
                    if ((item >> 2) < b_rows) pk[i] = lds128(src + (item >> 2) * PK_ROW + (item & 3) * 16);
                }
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    const int item = t + i * kUnpackGroup * 32;
                    const int r = item >> 2, c = item & 3;
                    if (r >= b_rows) continue;
                    uint4 lo, hi;
                    unpack_x16(pk[i], lo, hi);
                    const uint32_t rowaddr = dst + r * U8_ROW;
                    sts128(rowaddr + (((2 * c) ^ (r & 7)) << 4), lo);
                    sts128(rowaddr + (((2 * c + 1) ^ (r & 7)) << 4), hi);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(map_to_cta(full + 8 * us, 0));
                    mbar_arrive(empty_p + 8 * ps);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the MMAs have read the other CTA's shared memory, and nobody arrives on it any more
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_acc, 512);
    }
    cluster_sync();  // neither CTA leaves before the other has released the pair's tensor memory
}
