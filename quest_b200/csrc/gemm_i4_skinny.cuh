// int4 x int4 GEMM with the dequantising epilogue for few activation rows (decoding, short prompts): the weights are the
// M side of the MMA.  Included by gemm_i4.cu inside namespace qb, before the host side.
//
//   D[weight row, token] = W[128 rows, K] . A[TN tokens, K]^T      tcgen05.mma kind::i8, M 128, N = TN, K 32
//
// With few tokens the layer is a stream over the packed weights.  The 128-row tile kernel puts the tokens on the M side:
// a CTA then unpacks 256 weight rows and 128 mostly empty token rows per stage, and its four MMAs take the time of full
// ones whatever M is.  Here a CTA owns `rows` <= 128 weight rows (any multiple of 8, chosen so that the CTAs fill the
// SMs evenly), unpacks only them, copies the tokens ready-made (int8 in operand order) with TMA, and a step costs
// little more than its weights' way through shared memory.  Where the rows alone leave SMs idle or K is long, the CTAs of
// a cluster split K and add their int32 sums through distributed shared memory: no global scratch, no counters.
#pragma once

namespace skinny {
constexpr int W_ROWS = 128;                     // rows of the MMA; a CTA uses the first `rows` of them
constexpr int kUnpackWarps = 8, kFirstUnpack = 2;
constexpr int kUnpackGroup = 4;                 // warps that unpack one stage; the two groups take turns
constexpr int kTokenWarp = kFirstUnpack + kUnpackWarps;
constexpr int kWarps = kTokenWarp + 1;
constexpr int kThreads = kWarps * 32;
constexpr int W_BYTES = W_ROWS * U8_ROW;        // int8 weights per stage
constexpr int P_BYTES = W_ROWS * PK_ROW;        // packed weights per stage
constexpr int kMaxSplit = 8;
template <int TN>
struct Cfg {
    // two CTAs per SM up to 32 tokens (at most 113 KB each), one beyond
    static constexpr int U_STAGES = TN <= 32 ? 3 : 4;
    static constexpr int T_STAGES = TN == 16 ? 8 : (TN == 128 || TN == 32 ? 4 : 6);
    static constexpr int P_STAGES = TN <= 32 ? 5 : (TN <= 64 ? 12 : 10);
    static constexpr int T_BYTES = TN * U8_ROW;
    static constexpr int NUM_BARS = 2 * P_STAGES + 2 * U_STAGES + 2 * T_STAGES + 1;
    static constexpr int RING_BYTES = U_STAGES * W_BYTES + T_STAGES * T_BYTES + P_STAGES * P_BYTES;
    static constexpr int SMEM_BYTES = 1024 + RING_BYTES + NUM_BARS * 8 + 16;
    static constexpr int TMEM_COLS = TN < 32 ? 32 : TN;
    static constexpr uint32_t IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(W_ROWS >> 4) << 24);
    static_assert(TN * W_ROWS * 4 <= RING_BYTES, "the sums are handed over in the rings");
};
}  // namespace skinny

// Grid: (tiles of `rows` weight rows) x S, in clusters of S along x: CTA blockIdx.x works on tile blockIdx.x / S and the
// K range of its rank in the cluster.
template <int TN>
__global__ void __launch_bounds__(skinny::kThreads)
gemm_i4_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_t,
                      const __grid_constant__ EpilogueParams ep, const int M, const int N, const int K, const int rows, const int S) {
    using namespace skinny;
    using C = skinny::Cfg<TN>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_base = smem_u32(smem_raw);
    const uint32_t smem_base = (raw_base + 1023u) & ~1023u;
    const uint32_t w_base = smem_base;                              // int8 weights, 128-byte swizzle
    const uint32_t t_base = w_base + C::U_STAGES * W_BYTES;         // tokens
    const uint32_t p_base = t_base + C::T_STAGES * C::T_BYTES;      // packed weights
    const uint32_t full_p = p_base + C::P_STAGES * P_BYTES;
    const uint32_t empty_p = full_p + 8 * C::P_STAGES;
    const uint32_t full = empty_p + 8 * C::P_STAGES;                // the weights are unpacked
    const uint32_t empty = full + 8 * C::U_STAGES;
    const uint32_t full_t = empty + 8 * C::U_STAGES;                // the tokens have landed
    const uint32_t empty_t = full_t + 8 * C::T_STAGES;
    const uint32_t done = empty_t + 8 * C::T_STAGES;                  // the accumulators are complete
    const uint32_t tmem_slot = done + 8;
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - raw_base));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // uniform, and known to be
    const int lane = threadIdx.x & 31;
    const int tile = S > 1 ? (int)blockIdx.x / S : (int)blockIdx.x;
    const int rank = S > 1 ? (int)blockIdx.x - tile * S : 0;
    const int n0 = tile * rows;
    const int num_kb = K / BK;
    const int kb0 = (int)((long long)num_kb * rank / S);
    const int steps = (int)((long long)num_kb * (rank + 1) / S) - kb0;  // at least one: the host keeps S <= num_kb
    const uint32_t p_bytes = (uint32_t)rows * PK_ROW;
    uint32_t pre_issued = 0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < C::P_STAGES; ++i) {
            mbar_init(full_p + 8 * i, 1);
            mbar_init(empty_p + 8 * i, kUnpackGroup);
        }
        for (int i = 0; i < C::U_STAGES; ++i) {
            mbar_init(full + 8 * i, kUnpackGroup);
            mbar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < C::T_STAGES; ++i) {
            mbar_init(full_t + 8 * i, 1);
            mbar_init(empty_t + 8 * i, 1);
        }
        mbar_init(done, 1);
        fence_barrier_init();
        tma_prefetch_desc(&tmap_w);
        // the first weight copies leave before tensor memory is allocated and the CTA has synchronised
        for (; pre_issued < (uint32_t)C::P_STAGES && (int)pre_issued < steps; ++pre_issued) {
            mbar_arrive_expect_tx(full_p + 8 * pre_issued, p_bytes);
            tma_load_2d(p_base + pre_issued * P_BYTES, &tmap_w, (kb0 + (int)pre_issued) * PK_ROW, n0, full_p + 8 * pre_issued);
        }
    }
    __syncwarp();
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_acc = *tmem_slot_ptr;
    let_dependents_launch();  // only now that tensor memory is allocated (see gemm_i4_kernel)

    if (warp == 0) {
        // ------------------------------ weight producer ------------------------------
        if (lane == 0) {
            uint32_t it = pre_issued;
            bool ok = true;
            for (; (int)it < steps; ++it) {
                const uint32_t s = it % C::P_STAGES, ph = (it / C::P_STAGES) & 1u;
                if (!(ok = mbar_wait(empty_p + 8 * s, ph ^ 1u, 51))) break;
                mbar_arrive_expect_tx(full_p + 8 * s, p_bytes);
                tma_load_2d(p_base + s * P_BYTES, &tmap_w, (kb0 + (int)it) * PK_ROW, n0, full_p + 8 * s);
            }
            const uint32_t pending = it < (uint32_t)C::P_STAGES ? it : (uint32_t)C::P_STAGES;
            for (uint32_t j = 0; j < pending; ++j) {  // do not go on while a copy of ours may still land
                const uint32_t i2 = it - 1 - j;
                mbar_wait(full_p + 8 * (i2 % C::P_STAGES), (i2 / C::P_STAGES) & 1u, 52);
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer (all lanes walk the loop, see elect_one) ------------------------
        const uint64_t dw0 = make_smem_desc(w_base), dt0 = make_smem_desc(t_base);
        uint32_t s = 0, ph = 0, st = 0, pht = 0;
        for (int it = 0; it < steps; ++it) {
            bool ok = mbar_wait(full_t + 8 * st, pht, 53) && mbar_wait(full + 8 * s, ph, 54);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint64_t dw = dw0 + (uint64_t)(s * (W_BYTES >> 4)), dt = dt0 + (uint64_t)(st * (C::T_BYTES >> 4));
            if (elect_one()) {
                umma_i8(tmem_acc, dw, dt, C::IDESC, it != 0 ? 1u : 0u);
#pragma unroll
                for (int j = 1; j < BK / 32; ++j) umma_i8(tmem_acc, dw + 2 * j, dt + 2 * j, C::IDESC, 1u);
                umma_commit(empty + 8 * s);
                umma_commit(empty_t + 8 * st);
            }
            __syncwarp();
            if (++s == C::U_STAGES) s = 0, ph ^= 1u;
            if (++st == C::T_STAGES) st = 0, pht ^= 1u;
        }
        if (elect_one()) umma_commit(done);  // on a give-up, too: the commit covers whatever was issued
        __syncwarp();
        mbar_wait(done, 0, 55);
        __syncwarp();
    } else if (warp == kTokenWarp) {
        // ------------------------------ token producer ------------------------------
        if (lane == 0) {
            tma_prefetch_desc(&tmap_t);
            wait_for_preceding_grid();  // the tokens are the quantiser's output
            uint32_t it = 0;
            for (; (int)it < steps; ++it) {
                const uint32_t st = it % C::T_STAGES, ph = (it / C::T_STAGES) & 1u;
                if (!mbar_wait(empty_t + 8 * st, ph ^ 1u, 58)) break;
                mbar_arrive_expect_tx(full_t + 8 * st, C::T_BYTES);
                tma_load_2d(t_base + st * C::T_BYTES, &tmap_t, (kb0 + (int)it) * U8_ROW, 0, full_t + 8 * st);
            }
            const uint32_t pending = it < (uint32_t)C::T_STAGES ? it : (uint32_t)C::T_STAGES;
            for (uint32_t j = 0; j < pending; ++j) {  // do not go on while a copy of ours may still land
                const uint32_t i2 = it - 1 - j;
                mbar_wait(full_t + 8 * (i2 % C::T_STAGES), (i2 / C::T_STAGES) & 1u, 59);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------ unpack warps ------------------------------
        const int grp = (warp - kFirstUnpack) / kUnpackGroup;
        const int t = (threadIdx.x - kFirstUnpack * 32) & (kUnpackGroup * 32 - 1);  // 0 .. 127
        for (int it = grp; it < steps; it += 2) {
            const uint32_t ps = (uint32_t)it % C::P_STAGES, pph = ((uint32_t)it / C::P_STAGES) & 1u;
            const uint32_t us = (uint32_t)it % C::U_STAGES, uph = ((uint32_t)it / C::U_STAGES) & 1u;
            // The parity of full_p names one phase only if the slot's use before (step it - P_STAGES) has ended: on an even ring
            // it was this group's own, on an odd one the MMAs of step it - 2 - U_STAGES, which this group has waited for, say so.
            static_assert(C::P_STAGES % 2 == 0 || C::U_STAGES + 2 <= C::P_STAGES, "a packed slot's use before this one has ended");
            bool ok = mbar_wait(full_p + 8 * ps, pph, 56) && mbar_wait(empty + 8 * us, uph ^ 1u, 57);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t src = p_base + ps * P_BYTES;
            const uint32_t dst = w_base + us * W_BYTES;
            constexpr int ITEMS = W_ROWS * 4 / (kUnpackGroup * 32);  // 4 pieces of 16 packed bytes per thread
            uint4 pk[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const int item = t + i * kUnpackGroup * 32;  // a warp covers eight rows: the row test is uniform
                if ((item >> 2) < rows) pk[i] = lds128(src + (item >> 2) * PK_ROW + (item & 3) * 16);
            }
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const int item = t + i * kUnpackGroup * 32;
                const int r = item >> 2, c = item & 3;
                if (r >= rows) continue;
                uint4 lo, hi;
                unpack_x16(pk[i], lo, hi);
                const uint32_t rowaddr = dst + r * U8_ROW;
                sts128(rowaddr + (((2 * c) ^ (r & 7)) << 4), lo);
                sts128(rowaddr + (((2 * c + 1) ^ (r & 7)) << 4), hi);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(full + 8 * us);
                mbar_arrive(empty_p + 8 * ps);
            }
        }
    }

    // All MMAs of this CTA have completed (the issuer waited for them) and all copies have landed: the rings are free.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Sums -> shared memory as [token][weight row]: four warps, one per tensor-memory lane quadrant.
    if (warp >= kFirstUnpack && warp < kFirstUnpack + 4) {
        const int quad = warp & 3;
        const uint32_t dst = smem_base + (uint32_t)(quad * 32 + lane) * 4u;
#pragma unroll 1
        for (int c0 = 0; c0 < TN && c0 < M; c0 += 16) {
            uint32_t r[16];
            tmem_ld16(tmem_acc + ((uint32_t)(quad * 32) << 16) + c0, r);
            tmem_ld_wait16(r);
#pragma unroll
            for (int i = 0; i < 16; ++i)
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (uint32_t)(c0 + i) * (W_ROWS * 4)), "r"(r[i]) : "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_acc, C::TMEM_COLS);
    }
    wait_for_preceding_grid();  // row sums and scales are the quantiser's output
    if (S > 1) cluster_sync();
    // Tokens rank, rank + S, ... of the tile: add the S partial sums, dequantise, store.  A warp covers 128 weight rows of
    // one token as 32 x 4 consecutive outputs.
    const bool vec = ep.vec_ok && (n0 & 3) == 0;
    const int c = lane * 4;
    if (c < rows) {
        int ba[4];
        float bm[4], bias[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool in = n0 + c + i < N;
            ba[i] = in ? ep.b_add[n0 + c + i] : 0;
            bm[i] = in ? bf16_to_f32(ep.b_mul[n0 + c + i]) : 0.f;
            bias[i] = in && ep.bias != nullptr ? bf16_to_f32(ep.bias[n0 + c + i]) : 0.f;
        }
        for (int m = rank + warp * S; m < M; m += kWarps * S) {
            const uint32_t src = smem_base + (uint32_t)(m * W_ROWS + c) * 4u;
            int acc[4] = {0, 0, 0, 0};
            for (int s = 0; s < S; ++s) {
                const uint32_t a = S > 1 ? map_to_cta(src, (uint32_t)s) : src;
                int v[4];
                if (S > 1) {
                    asm volatile("ld.shared::cluster.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a) : "memory");
                } else {
                    asm volatile("ld.shared.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a) : "memory");
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i] += v[i];  // multiples of 256, |sum| < 2^31 (K < 2^17)
            }
            const int a_add = ep.a_add[m];
            const float am = 0.5f * bf16_to_f32(ep.a_mul[m]);
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = (float)((acc[i] >> 7) + a_add + ba[i]) * (am * bm[i]);
            __nv_bfloat16* out = static_cast<__nv_bfloat16*>(ep.out) + (size_t)m * ep.ld + n0 + c;
            uint32_t w0 = pack_bf16x2(v[0], v[1]), w1 = pack_bf16x2(v[2], v[3]);
            if (ep.bias != nullptr) {
                w0 = pack_bf16x2(bf16lo_to_f32(w0) + bias[0], bf16hi_to_f32(w0) + bias[1]);
                w1 = pack_bf16x2(bf16lo_to_f32(w1) + bias[2], bf16hi_to_f32(w1) + bias[3]);
            }
            if (vec && n0 + c + 4 <= N) {
                *reinterpret_cast<uint2*>(out) = make_uint2(w0, w1);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (n0 + c + i < N) reinterpret_cast<uint16_t*>(out)[i] = (uint16_t)((i < 2 ? w0 : w1) >> (16 * (i & 1)));
            }
        }
    }
    if (S > 1) cluster_sync();  // the other CTAs have read this one's sums
}
