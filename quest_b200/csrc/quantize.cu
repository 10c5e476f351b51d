// Row-wise kernels of the W4A4 linear path for sm_100a:
//   - fused block-Hadamard + RMS scale + int4 quantise + pack + row-sum (one pass over x),
//   - the reference's unfused find_scale_int4 / quantize_int4 (same kernel, other template arms),
//   - add_mul_vv (the exact dequantising epilogue as a standalone kernel).
//
// All of them are HBM-bandwidth bound.  One thread block owns one row; every lane owns runs of 32
// contiguous elements (four 16-byte loads, one 16-byte packed store), a "unit" being the 1024
// elements a warp covers at once.  The whole row stays in registers (as bf16 pairs) between the
// sum-of-squares pass and the quantise pass, so x is read from HBM exactly once.
//
// Numerics follow gemm-quest/quest/quantize_kernel.cu and gemm-quest/benchmarks/utils.py:
//   two rounding points decide the codes - the Hadamard output is rounded to bf16 before anything
//   else looks at it, and the scale is rounded to bf16 before the divide.
#include "common.cuh"
#include "hadamard_unit.cuh"
#include "tcgen05.cuh"

namespace qb {

thread_local bool qb_tl_dependent_quantiser = false;
thread_local bool qb_tl_in_layer = false;
thread_local int qb_tl_quantiser_kernel = 0;

struct RowParams {
    const __nv_bfloat16* x;        // [M,K] input
    __nv_bfloat16* x_out;          // optional [M,K] output (transformed or dequantised values)
    const __nv_bfloat16* scale_in; // optional [M] scale to quantise with
    __nv_bfloat16* scale_out;      // optional [M] computed scale
    int8_t* q_dense;               // optional [M,K]
    uint8_t* q_packed;             // optional [M,K/2]
    uint8_t* q_a8;                 // optional [M,K]: sixteen times the codes as int8, in the GEMM's operand order (instead of q_packed)
    int32_t* row_sum;              // optional [M]
    int K;
    int M;
    const __nv_bfloat16* x2;       // producer-fused kernels: second input [M,K] (the "up" branch of SiLU(gate) * up)
    const __nv_bfloat16* norm_w;   // producer-fused kernels: RMSNorm weight [K]
    float norm_eps;                // RMSNorm epsilon
    float had_scale;               // Hadamard normalisation constant
    int x_out_mode;                // 0 none, 1 transformed values, 2 dequantised values
    int quantize;                  // 0: stop after the scale (find_scale / transform only)
    int row_sum_add;               // row_kernel only: constant added to every row sum
    int let_dependents;            // inside a layer: the GEMM behind this kernel may be scheduled early (1: at once, 2: when a
                                   // block has done its last rows; mma.sync kernel only).  Never otherwise: what
                                   // is written here may be the weights of a layer further on, whose GEMM reads its first
                                   // weights before it waits.
};

constexpr int kMaxVectorK = 64 * kUnit;  // 16 warps x 4 units; longer rows take the scalar kernel
// floor(x / s) for bf16-valued x and s, without a divide.
//
// x / s is an exact integer for about 1 % of the elements, so a plain x * (1/s) mis-floors.  For
// bf16 operands every non-integer quotient of magnitude <= 8 is at least 2^-9 away from an integer,
// while x * rcp(s) is within 2^-22 relative of the true quotient; nudging the product by
// |y| * 2^-13 towards +inf therefore lands exact integers on or above themselves and moves nothing
// else across an integer (and keeps the sign of tiny quotients, so -tiny still floors to -1).
// Verified exhaustively over all pairs of bf16 mantissas and the exponent differences that matter.
// Returns floor as an int; out-of-range quotients keep their sign and saturate later.
__device__ __forceinline__ int floor_quotient(float x, float inv_s) {
    const float y = x * inv_s;
    const float y2 = fmaf(fabsf(y), 1.220703125e-4f, y);
    return __float_as_int(__fadd_rd(y2, kFloorMagic)) - kFloorMagicBits;
}

// (sat4(a) << 4 | sat4(b)) | (c << 8): saturating pack of two int32 to signed nibbles.
__device__ __forceinline__ uint32_t pack_sat_s4(int hi, int lo, uint32_t c) {
    uint32_t d;
    asm("cvt.pack.sat.s4.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(hi), "r"(lo), "r"(c));
    return d;
}

// 32 packed codes as the GEMM's int8 operand: sixteen times the codes, the even positions of the group first (see q_a8).
__device__ __forceinline__ void store_a8(uint8_t* dst, const uint4& w) {
    *reinterpret_cast<uint4*>(dst) = make_uint4((w.x << 4) & 0xF0F0F0F0u, (w.y << 4) & 0xF0F0F0F0u, (w.z << 4) & 0xF0F0F0F0u, (w.w << 4) & 0xF0F0F0F0u);
    *reinterpret_cast<uint4*>(dst + 16) = make_uint4(w.x & 0xF0F0F0F0u, w.y & 0xF0F0F0F0u, w.z & 0xF0F0F0F0u, w.w & 0xF0F0F0F0u);
}

template <int HB>
__device__ __forceinline__ void hadamard32(float (&f)[32], int lane) {
    // Index bits 0..4 live in registers.
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if ((i & s) == 0) {
                const float a = f[i], b = f[i + s];
                f[i] = a + b;
                f[i + s] = a - b;
            }
        }
    }
    // The remaining log2(HB/32) index bits are lane bits: butterfly through warp shuffles.
#pragma unroll
    for (int m = 1; m < HB / 32; m <<= 1) {
        const float sgn = (lane & m) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const float p = __shfl_xor_sync(0xffffffffu, f[i], m);
            f[i] = fmaf(f[i], sgn, p);  // lower lane: a + b, upper lane: a - b
        }
    }
}

// HB: Hadamard block (0 = none).  UNITS: 1024-element units per warp.  EXTRAS: compile the rarely
// used outputs (dense int8 codes, transformed / dequantised bf16 values).
template <int HB, int UNITS, bool EXTRAS>
__global__ void __launch_bounds__(UNITS == 1 ? 256 : 512) row_kernel(const RowParams p) {
    if (!EXTRAS && p.let_dependents) let_dependents_launch();
    const int row = blockIdx.x;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const int K = p.K;
    const __nv_bfloat16* xr = p.x + (size_t)row * K;

    __shared__ double red_f[32];
    __shared__ int red_i[32];

    uint32_t v[UNITS][16];  // the lane's elements as bf16 pairs, after the transform
    float ssq = 0.f;

    // Issue every load of the row before touching the data.
    uint4 raw[UNITS][4];
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        const int e0 = (u * nwarps + warp) * kUnit + lane * 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            raw[u][j] = make_uint4(0, 0, 0, 0);
            if (e0 + 8 * j < K) {
                // The EXTRAS arms may write x in place, so they use ordinary (coherent) loads.
                if (EXTRAS) raw[u][j] = *reinterpret_cast<const uint4*>(xr + e0 + 8 * j);
                else raw[u][j] = ld_stream16(xr + e0 + 8 * j);
            }
        }
    }

#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(&raw[u][0]);
        if (HB > 0) {
            float f[32];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                f[2 * i] = bf16lo_to_f32(w[i]);
                f[2 * i + 1] = bf16hi_to_f32(w[i]);
            }
            hadamard32<HB>(f, lane);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[u][i] = pack_bf16x2(f[2 * i] * p.had_scale, f[2 * i + 1] * p.had_scale);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[u][i] = w[i];
        }
        if (p.scale_in == nullptr) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float a = bf16lo_to_f32(v[u][i]), b = bf16hi_to_f32(v[u][i]);
                ssq = fmaf(a, a, ssq);
                ssq = fmaf(b, b, ssq);
            }
        }
    }

    // ---- scale ----
    float s;
    if (p.scale_in != nullptr) {
        s = bf16_to_f32(p.scale_in[row]);
    } else {
        double t = (double)ssq;
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) t += __shfl_xor_sync(0xffffffffu, t, m);
        if (lane == 0) red_f[warp] = t;
        __syncthreads();
        double tot = 0.0;
        for (int i = 0; i < nwarps; ++i) tot += red_f[i];
        const float mean_sq = (float)(tot / (double)K);
        const __nv_bfloat16 sb = __float2bfloat16_rn(quest_scale_from_mean_square(mean_sq));
        if (threadIdx.x == 0 && p.scale_out != nullptr) p.scale_out[row] = sb;
        s = bf16_to_f32(sb);
    }

    if (EXTRAS && p.x_out_mode == 1) {
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int e0 = (u * nwarps + warp) * kUnit + lane * 32;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (e0 + 8 * j < K)
                    *reinterpret_cast<uint4*>(p.x_out + (size_t)row * K + e0 + 8 * j) =
                        make_uint4(v[u][4 * j], v[u][4 * j + 1], v[u][4 * j + 2], v[u][4 * j + 3]);
        }
    }
    if (!p.quantize) return;

    // ---- quantise, pack, row sum ----
    const float inv_s = __frcp_rn(s);
    const bool vec_store = (K & 31) == 0;
    int rs16 = 0;
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        const int e0 = (u * nwarps + warp) * kUnit + lane * 32;
        uint32_t pk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int q[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                q[2 * i] = floor_quotient(bf16lo_to_f32(v[u][4 * j + i]), inv_s);
                q[2 * i + 1] = floor_quotient(bf16hi_to_f32(v[u][4 * j + i]), inv_s);
            }
            uint32_t d = pack_sat_s4(q[7], q[6], 0u);
            d = pack_sat_s4(q[5], q[4], d);
            d = pack_sat_s4(q[3], q[2], d);
            d = pack_sat_s4(q[1], q[0], d);
            pk[j] = d;
            rs16 = nibble_sum16(d, rs16);  // padding lanes hold zeros: code 0, adds nothing

            if (EXTRAS && e0 + 8 * j < K) {
                if (p.q_dense != nullptr) {
                    uint32_t lo = 0, hi = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        lo |= (uint32_t)(min(max(q[i], -8), 7) & 0xFF) << (8 * i);
                        hi |= (uint32_t)(min(max(q[4 + i], -8), 7) & 0xFF) << (8 * i);
                    }
                    *reinterpret_cast<uint2*>(p.q_dense + (size_t)row * K + e0 + 8 * j) = make_uint2(lo, hi);
                }
                if (p.x_out_mode == 2) {
                    uint32_t o[4];
                    const float half_s = s * 0.5f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float a = fmaf((float)min(max(q[2 * i], -8), 7), s, half_s);
                        const float b = fmaf((float)min(max(q[2 * i + 1], -8), 7), s, half_s);
                        o[i] = pack_bf16x2(a, b);
                    }
                    *reinterpret_cast<uint4*>(p.x_out + (size_t)row * K + e0 + 8 * j) =
                        make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
        }
        if (!EXTRAS && p.q_a8 != nullptr) {  // K is a multiple of 128 here
            if (e0 < K) store_a8(p.q_a8 + (size_t)row * K + e0, make_uint4(pk[0], pk[1], pk[2], pk[3]));
        } else if (p.q_packed != nullptr) {
            uint8_t* dst = p.q_packed + (size_t)row * (K >> 1) + (e0 >> 1);
            if (vec_store) {
                if (e0 < K) *reinterpret_cast<uint4*>(dst) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (e0 + 8 * j < K) *reinterpret_cast<uint32_t*>(dst + 4 * j) = pk[j];
            }
        }
    }
    if (p.row_sum != nullptr) {
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) rs16 += __shfl_xor_sync(0xffffffffu, rs16, m);
        if (lane == 0) red_i[warp] = rs16;
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int i = 0; i < nwarps; ++i) tot += red_i[i];
            p.row_sum[row] = (tot >> 4) + p.row_sum_add;  // exact: every term is a multiple of 16
        }
    }
}

// -------------------------------------------------------------------------------------------------
// The hot path: fused Hadamard + scale + quantise + pack + row sum, tensor-core assisted.
//
// The shuffle-butterfly kernel above spends ~26 instructions per element and is issue-bound at well
// under half of the HBM bandwidth.  Here the block transform is factored as H_block = H_a (x) H_16:
// the 16-point factor over the low four index bits is a tiny bf16 MMA (mma.sync m16n8k16, A = sixteen
// contiguous activations per row, B = +-bf16(block^-0.5) Sylvester signs, fp32 accumulate - the same
// "x times Hadamard matrix" product the reference hands to cuBLAS), and the factor over the high index
// bits is a butterfly over values a thread already holds.  Data path per warp and 1024 elements:
//   cp.async 16 B/lane global -> warp-private shared memory (blocks padded to 272 B: conflict-free)
//   ldmatrix x4  -> A fragments, 8 MMAs -> 32 fp32 values per thread (8 high-index rows x 4 columns)
//   butterflies, round to bf16 pairs (kept in registers until the row's scale is known)
//   quantise -> 2-byte pieces -> warp-private shared staging -> one coalesced 16-byte store per lane.
// -------------------------------------------------------------------------------------------------
constexpr int kMaxDynSmem = 220 * 1024;  // leaves room for the static reduction arrays under the 227 KB limit
constexpr int kStepBytes = 2 * kStepIn;  // two input buffers (the next row is prefetched); the packed codes are
                                         // staged in the buffer that has just been consumed

// Thread-block shape: G row groups x W warps.  The W warps of a group share one row (UNITS 1024-element
// units per warp); the block walks over batches of G rows.  Everything that is per row rather than per
// element (summing the partial sums, sqrt, rounding the scale, its reciprocal, the clamp bounds) is a short
// float chain that every warp evaluates for its own row right after the one barrier that publishes the partial
// sums; the final row sums are written one batch later by warp 0.
#ifdef QB200_TRACE
// Tuning builds only: earliest block start, latest start, earliest end and latest end (globaltimer, ns) of the last launch.
__device__ unsigned long long g_hq_trace[6] = {~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull};  // [4], [5]: first accumulator ready (tcgen05 kernel)
__device__ __forceinline__ unsigned long long hq_gtime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#endif

// PRO: what produces the rows that are transformed and quantised.
//   0  the input itself.
//   1  RMSNorm of the input:  y = bf16( bf16(x * rsqrt(mean(x^2) + eps)) * w )   (src/models/llama.py:64-76: the
//      normalised value is cast back to the activation type before the weight multiplies it).
//   3  the residual add in front of the norm as well: x + x2 is rounded to bf16, written to x_out (which may be x2) and
//      normalised as in 1.
//   2  SwiGLU gate:           y = bf16( bf16(silu(x)) * x2 ),  silu(x) = x / (1 + exp(-x)) in fp32
//      (src/models/llama.py:118, torch's silu for bf16 inputs).
// The producer rewrites the row in shared memory, in place, between the copy and the tensor-core stage; everything
// after it is unchanged.  It saves the producer's own kernel(s), one write and one read of [M, K] bf16.
constexpr int kProNone = 0, kProRmsNorm = 1, kProSiluMul = 2, kProAddRmsNorm = 3;

// silu of eight bf16 values, rounded to bf16 as the correctly rounded fp32 quotient x / (1 + exp(-x)) is: the product with
// the approximate reciprocal is within 3 ulp of the quotient, which matters only within 4 ulp of a tie between two bf16
// values (one in 7000); there, and for divisors whose reciprocal comes near the subnormal range, the chunk is divided in
// full.  One branch per eight values.
__device__ __forceinline__ void silu8(const uint32_t (&w)[4], uint32_t (&t)[4]) {
    float d[8], q[8];
    bool exact = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float a = (i & 1) ? bf16hi_to_f32(w[i / 2]) : bf16lo_to_f32(w[i / 2]);
        d[i] = 1.f + expf(-a);
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d[i]));  // d >= 1
        q[i] = a * r;
        exact |= (__float_as_uint(q[i]) & 0xFFFFu) - 0x7FFCu <= 8u || !(d[i] < 1e30f);
    }
    if (exact) {
#pragma unroll
        for (int i = 0; i < 8; ++i) q[i] = __fdiv_rn((i & 1) ? bf16hi_to_f32(w[i / 2]) : bf16lo_to_f32(w[i / 2]), d[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = pack_bf16x2(q[2 * i], q[2 * i + 1]);
}

// A8: writes the GEMM's int8 operand (q_a8, K a multiple of 128) instead of packed codes.  A template parameter: as a run-time
// test in the store loop it cost the packed form registers and 6 to 8 % (K 5632, 268 M elements, block 64: 185 -> 200 us).
template <int HB, int UNITS, int PRO = kProNone, bool A8 = false>
__global__ void __launch_bounds__(256, UNITS == 1 ? 4 : (UNITS == 2 ? 3 : 2))
hadamard_quant_mma_kernel(const RowParams p, const int W, const int G, const int nbuf) {
    extern __shared__ __align__(16) uint8_t hq_smem[];
    __shared__ float part_ssq[2][8];  // indexed by batch parity: one barrier per batch is enough
    __shared__ int part_rs[2][8];
    __shared__ float part_norm[8];    // PRO == kProRmsNorm: the warps' partial sums of squares of the raw row

#ifdef QB200_TRACE
    if (threadIdx.x == 0) {
        const unsigned long long t = hq_gtime();
        atomicMin(&g_hq_trace[0], t);
        atomicMax(&g_hq_trace[1], t);
    }
#endif
    // A kernel launched behind this one with a programmatic dependency (the GEMM of the layer call) may start its own
    // prologue now; it waits for this grid's results itself.
    if (p.let_dependents == 1) let_dependents_launch();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int grp = warp / W;      // row group of this warp
    const int wig = warp - grp * W;  // warp index within the group
    const int g = lane >> 2, tig = lane & 3;
    const int K = p.K, M = p.M;
    // nbuf = 2: the next row's copies are in flight while this row is processed.  nbuf = 1 (every row batch of the
    // launch is resident at once, nothing to prefetch): half the shared memory, twice the blocks per SM.
    const int step_bytes = nbuf * kStepIn;
    const uint32_t smem_w = (uint32_t)__cvta_generic_to_shared(hq_smem) + warp * (UNITS * step_bytes);
    const int num_batches = (M + G - 1) / G;

    // Copies of this warp's units of one row into input buffer `buf` (16 bytes per lane and instruction).
    auto issue_row = [&](int row, int buf) {
        if (row < M) {
            const __nv_bfloat16* xr = p.x + (size_t)row * K;
#pragma unroll
            for (int u = 0; u < UNITS; ++u) {
                const int unit = u * W + wig;
                const uint32_t in_base = smem_w + u * step_bytes + buf * kStepIn;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = j * 32 + lane;  // 16-byte chunk within the unit
                    const int e = unit * kUnit + c * 8;
                    const bool valid = e < K;
                    cp_async16_zfill(in_base + (c >> 4) * kBlkPitch + (c & 15) * 16,
                                     valid ? (const void*)(xr + e) : (const void*)xr, valid);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    int batch = blockIdx.x;
    if (batch < num_batches) issue_row(batch * G + grp, 0);

    // ---- B fragments: h * H16[k][o], MMA column n of tile nu is output o = 4*(n>>1) + 2*nu + (n&1) ----
    uint32_t bfrag[2][2];
    hadamard16_fragments(p.had_scale, lane, bfrag);

    int prev_batch = -1, last_par = 0;
    for (int it = 0; batch < num_batches; batch += gridDim.x, ++it) {
        const int buf = nbuf == 2 ? (it & 1) : 0;
        const int row = batch * G + grp;
        const int next = batch + gridDim.x;
        if (nbuf == 2 && next < num_batches) {
            issue_row(next * G + grp, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            if (nbuf == 1 && it > 0) issue_row(row, 0);  // single buffer: fetch this row now (the staging reads are done)
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();

        if (PRO != kProNone) {
            // Each lane owns the 16-byte chunks it copied itself (chunk c = 32 j + lane of every unit).
            constexpr bool kNorm = PRO == kProRmsNorm || PRO == kProAddRmsNorm;
            float rinv = 0.f;
            if (kNorm) {
                float nsq = 0.f;
#pragma unroll
                for (int u = 0; u < UNITS; ++u) {
                    const uint32_t in_base = smem_w + u * step_bytes + buf * kStepIn;
                    uint4 in2[4];
                    if (PRO == kProAddRmsNorm) {  // a unit's pieces are requested together
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int e = (u * W + wig) * kUnit + (j * 32 + lane) * 8;
                            if (e < K && row < M) in2[j] = *reinterpret_cast<const uint4*>(p.x2 + (size_t)row * K + e);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c = j * 32 + lane;
                        const uint32_t addr = in_base + (c >> 4) * kBlkPitch + (c & 15) * 16;
                        const uint4 q = lds128(addr);  // zero beyond K
                        uint32_t w4[4] = {q.x, q.y, q.z, q.w};
                        const int e = (u * W + wig) * kUnit + c * 8;
                        if (PRO == kProAddRmsNorm && e < K && row < M) {
                            const uint4 o = in2[j];
                            const uint32_t o4[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                w4[i] = pack_bf16x2(bf16lo_to_f32(w4[i]) + bf16lo_to_f32(o4[i]), bf16hi_to_f32(w4[i]) + bf16hi_to_f32(o4[i]));
                            const uint4 sum = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                            *reinterpret_cast<uint4*>(p.x_out + (size_t)row * K + e) = sum;
                            sts128(addr, sum);
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float a = bf16lo_to_f32(w4[i]), b = bf16hi_to_f32(w4[i]);
                            nsq = fmaf(a, a, nsq);
                            nsq = fmaf(b, b, nsq);
                        }
                    }
                }
#pragma unroll
                for (int m2 = 16; m2 > 0; m2 >>= 1) nsq += __shfl_xor_sync(0xffffffffu, nsq, m2);
                if (W > 1) {  // block-uniform: the row is spread over W warps
                    if (lane == 0) part_norm[warp] = nsq;
                    __syncthreads();
                    nsq = 0.f;
                    for (int i = 0; i < W; ++i) nsq += part_norm[grp * W + i];
                    __syncthreads();  // part_norm is rewritten for the next batch
                }
                rinv = rsqrtf(__fdiv_rn(nsq, (float)K) + p.norm_eps);
            }
            const int row_p = batch * G + grp;
#pragma unroll
            for (int u = 0; u < UNITS; ++u) {
                const int unit = u * W + wig;
                const uint32_t in_base = smem_w + u * step_bytes + buf * kStepIn;
                uint4 in2[4];
                if (PRO == kProSiluMul) {  // a unit's pieces are requested together, before the first is used
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = unit * kUnit + (j * 32 + lane) * 8;
                        if (e < K && row_p < M) in2[j] = ld_stream16(p.x2 + (size_t)row_p * K + e);
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = j * 32 + lane;
                    const int e = unit * kUnit + c * 8;
                    if (e >= K || row_p >= M) continue;
                    const uint32_t addr = in_base + (c >> 4) * kBlkPitch + (c & 15) * 16;
                    const uint4 q = lds128(addr);
                    const uint4 o = kNorm ? __ldg(reinterpret_cast<const uint4*>(p.norm_w + e)) : in2[j];
                    const uint32_t w4[4] = {q.x, q.y, q.z, q.w}, o4[4] = {o.x, o.y, o.z, o.w};
                    uint32_t t4[4], y4[4];  // t4: the producer's first rounding to the activation type
                    if (kNorm) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) t4[i] = pack_bf16x2(bf16lo_to_f32(w4[i]) * rinv, bf16hi_to_f32(w4[i]) * rinv);
                    } else {
                        silu8(w4, t4);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        y4[i] = pack_bf16x2(bf16lo_to_f32(t4[i]) * bf16lo_to_f32(o4[i]), bf16hi_to_f32(t4[i]) * bf16hi_to_f32(o4[i]));
                    sts128(addr, make_uint4(y4[0], y4[1], y4[2], y4[3]));
                }
            }
            __syncwarp();  // ldmatrix below reads chunks written by other lanes of this warp
        }

        uint32_t v[UNITS][16];  // v[u][2a + nu]: elements 16a + 4tig + 2nu (+1) of block g of the unit
        f32x2 ssq2 = 0ull;
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            transform_unit<HB>(smem_w + u * step_bytes + buf * kStepIn, lane, bfrag, v[u], ssq2);
        }
        float ssq;
        {
            float s0, s1;
            unpk2(ssq2, s0, s1);
            ssq = s0 + s1;
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, m);
        const int par = it & 1;
        if (lane == 0) part_ssq[par][warp] = ssq;
        __syncthreads();  // the partial sums of this batch (and the row-sum partials of the previous one) are in place

        // Every warp derives its row's constants itself (a short float chain, W partial sums): no second barrier
        // and nobody waits for a designated warp.  Warp 0 additionally publishes the scales and finishes the row
        // sums of the previous batch, off everyone's critical path.
        double tot = 0.0;
        for (int i = 0; i < W; ++i) tot += (double)part_ssq[par][grp * W + i];
        const __nv_bfloat16 sb = __float2bfloat16_rn(quest_scale_from_mean_square(__fdiv_rn((float)tot, (float)K)));
        const RowConstants rc = row_constants(sb);
        if (wig == 0 && lane == 0 && row < M) p.scale_out[row] = sb;
        if (warp == 0 && lane < G && prev_batch >= 0 && p.row_sum != nullptr) {
            const int pr = prev_batch * G + lane;
            if (pr < M) {
                int t2 = 0;
                for (int i = 0; i < W; ++i) t2 += part_rs[par ^ 1][lane * W + i];
                p.row_sum[pr] = t2 >> 4;  // exact: every term is a multiple of 16
            }
        }

        // ---- quantise, stage, store ----
        const bool vec_store = (K & 31) == 0;
        int rs16 = 0;
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int unit = u * W + wig;
            const uint32_t out_base = smem_w + u * step_bytes + buf * kStepIn;  // input already consumed
            const uint4 w = quantise_unit(v[u], rc, out_base, lane, rs16);
            const int e0 = unit * kUnit + lane * 32;
            if (A8) {
                if (row < M && e0 < K) store_a8(p.q_a8 + (size_t)row * K + e0, w);
            } else if (row < M) {
                uint8_t* dst = p.q_packed + (size_t)row * (K >> 1) + (e0 >> 1);
                if (vec_store) {
                    if (e0 < K) *reinterpret_cast<uint4*>(dst) = w;
                } else {
                    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (e0 + 8 * j < K) *reinterpret_cast<uint32_t*>(dst + 4 * j) = ww[j];
                }
            }
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) rs16 += __shfl_xor_sync(0xffffffffu, rs16, m);
        if (lane == 0) part_rs[par][warp] = rs16;
        prev_batch = batch;
        last_par = par;
    }
    // row sums of the last batch
    if (p.let_dependents == 2) let_dependents_launch();
    __syncthreads();
#ifdef QB200_TRACE
    if (threadIdx.x == 0) {
        const unsigned long long t = hq_gtime();
        atomicMin(&g_hq_trace[2], t);
        atomicMax(&g_hq_trace[3], t);
    }
#endif
    if (warp == 0 && lane < G && prev_batch >= 0 && p.row_sum != nullptr) {
        const int pr = prev_batch * G + lane;
        if (pr < M) {
            int t2 = 0;
            for (int i = 0; i < W; ++i) t2 += part_rs[last_par][lane * W + i];
            p.row_sum[pr] = t2 >> 4;
        }
    }
}

template <int HB, bool EXTRAS>
static int launch_row(const RowParams& p, cudaStream_t stream);

template <int HB, int PRO = kProNone>
static int launch_hq_mma(const RowParams& p_in, cudaStream_t stream) {
    RowParams p = p_in;
    if (p.let_dependents && (long long)p.M * p.K >= kTcFromInLayer) p.let_dependents = 2;
    const int units = (p.K + kUnit - 1) / kUnit;
    // units per warp, warps per row, rows per block (at most 16 warps per block)
    int per = units >= 2 ? 2 : 1;  // two units per warp amortise the per-row work best (measured)
    if (per > units) per = units;
    if (per != 1 && per != 2 && per != 4) per = 2;
    int W = (units + per - 1) / per;
    if (W > 8 && per < 4) { per = 4; W = (units + per - 1) / per; }
    if (W > 8) return PRO != kProNone ? QB200_ERR_UNSUPPORTED : launch_row<HB, false>(p, stream);  // very long rows: shuffle-butterfly kernel
    // Rows per block: up to 8 warps per block, but few rows overall want small blocks so that every SM ends
    // at the same time (a block is the unit the rows are dealt out in).
    int G = 8 / W;
    if (G < 1) G = 1;
    while (G > 1 && (long long)p.M < 96LL * 148 * G) G >>= 1;
    if (G > p.M) G = p.M;
    const int warps = W * G;
    const long long batches = ((long long)p.M + G - 1) / G;
    if ((size_t)warps * per * kStepBytes > kMaxDynSmem) return PRO != kProNone ? QB200_ERR_UNSUPPORTED : launch_row<HB, false>(p, stream);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess) return QB200_ERR_CUDA;
    {
        static int cached[64] = {0};
        if (dev >= 0 && dev < 64 && cached[dev] > 0) sms = cached[dev];
        else if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0) {
            if (dev >= 0 && dev < 64) cached[dev] = sms;
        } else sms = 148;
    }
    // Persistent grid: as many blocks as fit on the device at once (bounded by the number of row batches).
    // The caches are per kernel instantiation (index `which`) and per device.
    static bool attr_done[6][64] = {{false}};
    static int occ_cache[6][64][9][2] = {{{{0}}}};
    auto launch = [&](auto kernel, int which) -> int {
        const bool dev_ok = dev >= 0 && dev < 64;
        if (!(dev_ok && attr_done[which][dev])) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem) != cudaSuccess) {
                cudaGetLastError();  // reported through the return value; do not leave it pending
                return QB200_ERR_CUDA;
            }
            if (dev_ok) attr_done[which][dev] = true;
        }
        auto occupancy = [&](int nb) {
            int occ = dev_ok ? occ_cache[which][dev][warps][nb - 1] : 0;
            if (occ <= 0) {
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 32 * warps, (size_t)warps * per * nb * kStepIn) != cudaSuccess || occ <= 0) {
                    cudaGetLastError();
                    occ = 1;
                }
                if (dev_ok) occ_cache[which][dev][warps][nb - 1] = occ;
            }
            return occ;
        };
        // If every row batch fits on the device at once there is nothing to prefetch: use one input buffer.
        int nbuf = 2;
        long long grid = (long long)sms * occupancy(2);
        if (batches > grid && batches <= (long long)sms * occupancy(1)) {
            nbuf = 1;
            grid = (long long)sms * occupancy(1);
        }
        if (grid > batches) grid = batches;
        // Always an ordinary launch: behind a programmatic dependency this small kernel measured slower (M = 16, K = N =
        // 4096, layers back to back: 16.6 instead of 13.5 us per layer); only the tcgen05 kernel is launched that way.
        if (launch_kernel_dep(false, kernel, grid, 32 * warps, (size_t)warps * per * nbuf * kStepIn, stream, p, W, G, nbuf) != cudaSuccess) {
            cudaGetLastError();
            return QB200_ERR_CUDA;
        }
        return launch_status();
    };
    if (p.q_a8 != nullptr) {
        if (per == 1) return launch(hadamard_quant_mma_kernel<HB, 1, PRO, true>, 3);
        if (per == 2) return launch(hadamard_quant_mma_kernel<HB, 2, PRO, true>, 4);
        return launch(hadamard_quant_mma_kernel<HB, 4, PRO, true>, 5);
    }
    if (per == 1) return launch(hadamard_quant_mma_kernel<HB, 1, PRO>, 0);
    if (per == 2) return launch(hadamard_quant_mma_kernel<HB, 2, PRO>, 1);
    return launch(hadamard_quant_mma_kernel<HB, 4, PRO>, 2);
}

// Any K, any alignment, no Hadamard: one block per row, scalar accesses.  Only used for shapes the
// vector kernel does not cover (K not a multiple of 8, misaligned base pointers, K > 65536).
__global__ void __launch_bounds__(256) row_kernel_generic(const RowParams p) {
    const int row = blockIdx.x;
    const int K = p.K;
    const __nv_bfloat16* xr = p.x + (size_t)row * K;
    __shared__ double red_f[8];
    __shared__ int red_i[8];
    __shared__ float s_sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float s;
    if (p.scale_in != nullptr) {
        s = bf16_to_f32(p.scale_in[row]);
    } else {
        double t = 0.0;
        for (int k = threadIdx.x; k < K; k += blockDim.x) {
            const float a = bf16_to_f32(xr[k]);
            t += (double)(a * a);
        }
        for (int m = 16; m > 0; m >>= 1) t += __shfl_xor_sync(0xffffffffu, t, m);
        if (lane == 0) red_f[warp] = t;
        __syncthreads();
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int i = 0; i < 8; ++i) tot += red_f[i];
            const __nv_bfloat16 sb = __float2bfloat16_rn(quest_scale_from_mean_square((float)(tot / (double)K)));
            if (p.scale_out != nullptr) p.scale_out[row] = sb;
            s_sh = bf16_to_f32(sb);
        }
        __syncthreads();
        s = s_sh;
    }
    if (!p.quantize) return;
    const float inv_s = __frcp_rn(s);
    int rs = 0;
    // Each thread owns pairs of columns so that it can emit whole packed bytes.
    for (int k = 2 * threadIdx.x; k < K; k += 2 * blockDim.x) {
        int q[2] = {0, 0};
        for (int i = 0; i < 2; ++i) {
            if (k + i < K) {
                q[i] = min(max(floor_quotient(bf16_to_f32(xr[k + i]), inv_s), -8), 7);
                rs += q[i];
                if (p.q_dense != nullptr) p.q_dense[(size_t)row * K + k + i] = (int8_t)q[i];
                if (p.x_out_mode == 2)
                    p.x_out[(size_t)row * K + k + i] = __float2bfloat16_rn(fmaf((float)q[i], s, s * 0.5f));
            }
        }
        if (p.q_packed != nullptr && k + 1 < K)
            p.q_packed[(size_t)row * (K >> 1) + (k >> 1)] = (uint8_t)((q[1] << 4) | (q[0] & 0xF));
    }
    if (p.row_sum != nullptr) {
        for (int m = 16; m > 0; m >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, m);
        if (lane == 0) red_i[warp] = rs;
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int i = 0; i < 8; ++i) tot += red_i[i];
            p.row_sum[row] = tot;
        }
    }
}

template <int HB, bool EXTRAS>
static int launch_row(const RowParams& p, cudaStream_t stream) {
    const int units = (p.K + kUnit - 1) / kUnit;
    const dim3 grid((unsigned)p.M);
    if (units <= 8) {
        row_kernel<HB, 1, EXTRAS><<<grid, 32 * units, 0, stream>>>(p);
    } else if (units <= 32) {
        row_kernel<HB, 2, EXTRAS><<<grid, 32 * ((units + 1) / 2), 0, stream>>>(p);
    } else if (units <= 64) {
        row_kernel<HB, 4, EXTRAS><<<grid, 32 * ((units + 3) / 4), 0, stream>>>(p);
    } else {
        return QB200_ERR_UNSUPPORTED;
    }
    return launch_status();
}

#include "hadamard_quant_tc.cuh"

int hq_tc_fetch_and_clear_device_status(int* out) { return fetch_and_clear_device_status(out); }

bool hq_tc_shape_ok(int K) {
    int T, P;
    return K % 128 == 0 && hq_tc_tiling(K, &T, &P);
}

static bool vector_path_ok(const RowParams& p) {
    if (p.K % 8 != 0 || p.K > kMaxVectorK) return false;
    if (!aligned16(p.x)) return false;
    if (p.x_out != nullptr && !aligned16(p.x_out)) return false;
    if (p.q_dense != nullptr && (reinterpret_cast<uintptr_t>(p.q_dense) & 7u)) return false;
    if (p.q_packed != nullptr && !aligned16(p.q_packed)) return false;
    if (p.q_a8 != nullptr && (!aligned16(p.q_a8) || p.K % 128 != 0)) return false;
    return true;
}

static int run_rows(const RowParams& p, int block, bool extras, cudaStream_t stream) {
    if (p.M == 0 || p.K == 0) return QB200_OK;
    if (!vector_path_ok(p)) {
        if (block != 0) return QB200_ERR_UNSUPPORTED;
        row_kernel_generic<<<(unsigned)p.M, 256, 0, stream>>>(p);
        return launch_status();
    }
    switch (block) {
        case 0: return extras ? launch_row<0, true>(p, stream) : launch_row<0, false>(p, stream);
        case 64: return extras ? launch_row<64, true>(p, stream) : launch_row<64, false>(p, stream);
        case 128: return extras ? launch_row<128, true>(p, stream) : launch_row<128, false>(p, stream);
        case 256: return extras ? launch_row<256, true>(p, stream) : launch_row<256, false>(p, stream);
        default: return QB200_ERR_UNSUPPORTED;
    }
}

// -------------------------------------------------------------------------------------------------
// add_mul_vv: D = bf16( float(2C + a_add[m] + b_add[n]) * (0.5f * a_mul[m] * b_mul[n]) )
// 6 bytes per element of HBM traffic; eight columns per thread when N allows 16-byte accesses.
// -------------------------------------------------------------------------------------------------
__device__ __forceinline__ float dequant_one(int c, int a_add, int b_add, float a_mul, float b_mul) {
    const float lhs = (float)(c * 2 + a_add + b_add);
    const float rhs = 0.5f * a_mul * b_mul;
    return lhs * rhs;
}

__global__ void __launch_bounds__(256) add_mul_vv_vec8_kernel(__nv_bfloat16* __restrict__ d,
                                                              const int32_t* __restrict__ a_add,
                                                              const __nv_bfloat16* __restrict__ a_mul,
                                                              const int32_t* __restrict__ b_add,
                                                              const __nv_bfloat16* __restrict__ b_mul,
                                                              const int32_t* __restrict__ c, int M, int N) {
    const int groups_per_row = N >> 3;
    const long long total = (long long)M * groups_per_row;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
         g += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(g / groups_per_row);
        const int col = (int)(g - (long long)row * groups_per_row) << 3;
        const int aa = a_add[row];
        const float am = bf16_to_f32(a_mul[row]);
        const int4 c0 = *reinterpret_cast<const int4*>(c + (size_t)row * N + col);
        const int4 c1 = *reinterpret_cast<const int4*>(c + (size_t)row * N + col + 4);
        const int4 b0 = *reinterpret_cast<const int4*>(b_add + col);
        const int4 b1 = *reinterpret_cast<const int4*>(b_add + col + 4);
        const uint4 bm = *reinterpret_cast<const uint4*>(b_mul + col);
        uint4 o;
        o.x = pack_bf16x2(dequant_one(c0.x, aa, b0.x, am, bf16lo_to_f32(bm.x)),
                          dequant_one(c0.y, aa, b0.y, am, bf16hi_to_f32(bm.x)));
        o.y = pack_bf16x2(dequant_one(c0.z, aa, b0.z, am, bf16lo_to_f32(bm.y)),
                          dequant_one(c0.w, aa, b0.w, am, bf16hi_to_f32(bm.y)));
        o.z = pack_bf16x2(dequant_one(c1.x, aa, b1.x, am, bf16lo_to_f32(bm.z)),
                          dequant_one(c1.y, aa, b1.y, am, bf16hi_to_f32(bm.z)));
        o.w = pack_bf16x2(dequant_one(c1.z, aa, b1.z, am, bf16lo_to_f32(bm.w)),
                          dequant_one(c1.w, aa, b1.w, am, bf16hi_to_f32(bm.w)));
        *reinterpret_cast<uint4*>(d + (size_t)row * N + col) = o;
    }
}

__global__ void __launch_bounds__(256) add_mul_vv_scalar_kernel(__nv_bfloat16* __restrict__ d,
                                                                const int32_t* __restrict__ a_add,
                                                                const __nv_bfloat16* __restrict__ a_mul,
                                                                const int32_t* __restrict__ b_add,
                                                                const __nv_bfloat16* __restrict__ b_mul,
                                                                const int32_t* __restrict__ c, int M, int N) {
    const long long total = (long long)M * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(i / N);
        const int col = (int)(i - (long long)row * N);
        d[i] = __float2bfloat16_rn(
            dequant_one(c[i], a_add[row], b_add[col], bf16_to_f32(a_mul[row]), bf16_to_f32(b_mul[col])));
    }
}

// One block of bf16 [rows, cols] (row stride ld_bytes in every buffer) copied from src to n_dst destinations with one
// launch: the small-M exchange of the column-sharded layer (the block a rank has computed goes into every peer's
// output, which is mapped into this address space: plain 16-byte peer stores).
struct CopyDsts {
    void* p[7];
};

__global__ void copy_block_kernel(const uint8_t* __restrict__ src, const CopyDsts dsts, const int n_dst, const int rows,
                                  const int chunks, const long long ld_bytes) {
    const int total = rows * chunks;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const int r = idx / chunks, c = idx - r * chunks;
        const long long off = (long long)r * ld_bytes + (long long)c * 16;
        const uint4 v = *reinterpret_cast<const uint4*>(src + off);
        for (int d = 0; d < n_dst; ++d) *reinterpret_cast<uint4*>(static_cast<uint8_t*>(dsts.p[d]) + off) = v;
    }
}

// RMSNorm of bf16 rows, y = bf16(bf16(x * rsqrt(mean x^2 + eps)) * w): one warp per row, the row read once into registers
// in pieces of 2048 elements (longer rows are read a second time, from L1 or L2).  HBM-bound, 4 bytes per element.
__global__ void __launch_bounds__(256) rmsnorm_kernel(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x,
                                                      const __nv_bfloat16* __restrict__ w, const int M, const int K, const float eps) {
    const int lane = threadIdx.x & 31;
    for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < M; row += gridDim.x * 8) {
        const __nv_bfloat16* xr = x + (size_t)row * K;
        uint4 held[8];
        double total = 0.0;  // of pieces summed in eight chains of eight: a longer fp32 chain loses bits from K = 4096 on
        for (int base = 0; base < K; base += 2048) {
            float part[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int e = base + (j * 32 + lane) * 8;
                held[j] = e < K ? *reinterpret_cast<const uint4*>(xr + e) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t v[4] = {held[j].x, held[j].y, held[j].z, held[j].w};
                part[j] = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float a = bf16lo_to_f32(v[i]), b = bf16hi_to_f32(v[i]);
                    part[j] = fmaf(b, b, fmaf(a, a, part[j]));
                }
            }
            total += (double)(((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7])));
        }
        float sum = (float)total;
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
        const float rinv = rsqrtf(__fdiv_rn(sum, (float)K) + eps);
        for (int base = 0; base < K; base += 2048) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int e = base + (j * 32 + lane) * 8;
                if (e >= K) continue;
                if (K > 2048) held[j] = *reinterpret_cast<const uint4*>(xr + e);
                const uint4 wv = __ldg(reinterpret_cast<const uint4*>(w + e));
                const uint32_t v[4] = {held[j].x, held[j].y, held[j].z, held[j].w}, u[4] = {wv.x, wv.y, wv.z, wv.w};
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t t = pack_bf16x2(bf16lo_to_f32(v[i]) * rinv, bf16hi_to_f32(v[i]) * rinv);
                    o[i] = pack_bf16x2(bf16lo_to_f32(t) * bf16lo_to_f32(u[i]), bf16hi_to_f32(t) * bf16hi_to_f32(u[i]));
                }
                *reinterpret_cast<uint4*>(y + (size_t)row * K + e) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
}

// -------------------------------------------------------------------------------------------------
// Rotary embedding of q and k where the fused projection has left them (columns [0, cols) of each qkv row), in place.
// HBM-bound: one read and one write of q and k, 4 bytes per element, against a dozen passes in fp32 of the eager form.
// The same roundings as the eager form: each product, the difference / sum and the conversion to bf16 are rounded once.
// One thread owns four consecutive pairs (16 bytes); the table row of a position (head_dim * 8 bytes at most) stays in L1.
// -------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) rope_inplace_kernel(__nv_bfloat16* __restrict__ x, const T* __restrict__ table,
                                                           const long long chunks, const int row_chunks, const int seq,
                                                           const long long ld, const int head_dim) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < chunks; i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / row_chunks;
        const int col = (int)(i - row * row_chunks) * 8;
        const T* t = table + (size_t)(row % seq) * head_dim + col % head_dim;  // (cos, sin) of the chunk's four pairs
        float cs[8];
        if (sizeof(T) == 4) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(t)), b = __ldg(reinterpret_cast<const float4*>(t) + 1);
            cs[0] = a.x; cs[1] = a.y; cs[2] = a.z; cs[3] = a.w; cs[4] = b.x; cs[5] = b.y; cs[6] = b.z; cs[7] = b.w;
        } else {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(t));
            const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) cs[2 * j] = bf16lo_to_f32(w[j]), cs[2 * j + 1] = bf16hi_to_f32(w[j]);
        }
        uint4* p = reinterpret_cast<uint4*>(x + row * ld + col);
        const uint4 v = *p;
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float x0 = bf16lo_to_f32(w[j]), x1 = bf16hi_to_f32(w[j]), c = cs[2 * j], s = cs[2 * j + 1];
            w[j] = pack_bf16x2(__fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)), __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c)));
        }
        *p = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

}  // namespace qb

// -------------------------------------------------------------------------------------------------
// C ABI
// -------------------------------------------------------------------------------------------------
using namespace qb;

#ifdef QB200_TRACE
extern "C" int quest_b200_hq_trace(unsigned long long* out) {
    if (cudaDeviceSynchronize() != cudaSuccess) return QB200_ERR_CUDA;
    if (cudaMemcpyFromSymbol(out, g_hq_trace, sizeof(unsigned long long) * 6) != cudaSuccess) return QB200_ERR_CUDA;
    const unsigned long long init[6] = {~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull};
    return cuda_status(cudaMemcpyToSymbol(g_hq_trace, init, sizeof(init)));
}
#endif

extern "C" int find_scale_int4_cuda_bf16(void* scale_ptr, const void* x_ptr, int group_size, int batch_size,
                                         cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (batch_size == 0) return QB200_OK;
    if (scale_ptr == nullptr || x_ptr == nullptr || group_size == 0) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    p.K = group_size;
    p.M = batch_size;
    p.quantize = 0;
    return run_rows(p, 0, false, stream);
}

extern "C" int quantize_int4_cuda_bf16(void* x_ptr, const void* scale_ptr, void* x_int_ptr, void* x_int_packed_ptr,
                                       void* x_int_row_sum_ptr, int group_size, int batch_size, int do_dequantize,
                                       cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (batch_size == 0 || group_size == 0) return QB200_OK;
    if (x_ptr == nullptr || scale_ptr == nullptr) return QB200_ERR_INVALID_ARGUMENT;
    if (x_int_packed_ptr != nullptr && (group_size & 1)) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.scale_in = static_cast<const __nv_bfloat16*>(scale_ptr);
    p.q_dense = static_cast<int8_t*>(x_int_ptr);
    p.q_packed = static_cast<uint8_t*>(x_int_packed_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.K = group_size;
    p.M = batch_size;
    p.quantize = 1;
    if (do_dequantize) {
        p.x_out = static_cast<__nv_bfloat16*>(x_ptr);
        p.x_out_mode = 2;
    }
    const bool extras = do_dequantize || x_int_ptr != nullptr;
    return run_rows(p, 0, extras, stream);
}


extern "C" int hadamard_quantize_int4_cuda_bf16(void* x_int_packed_ptr, void* scale_ptr, void* x_int_row_sum_ptr,
                                                const void* x_ptr, int group_size, int batch_size, int block,
                                                cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (x_int_packed_ptr == nullptr || scale_ptr == nullptr || x_ptr == nullptr || group_size == 0)
        return QB200_ERR_INVALID_ARGUMENT;
    if (group_size % block != 0) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    p.q_packed = static_cast<uint8_t*>(x_int_packed_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.K = group_size;
    p.M = batch_size;
    p.quantize = 1;
    p.had_scale = __bfloat162float(__float2bfloat16_rn((float)(1.0 / sqrt((double)block))));
    p.let_dependents = qb_tl_in_layer;
    if (!vector_path_ok(p)) return QB200_ERR_UNSUPPORTED;
    // Tensor-core kernel where the shape fits its tiling; QB200_HQ_KERNEL=mma|tc forces one (tests, tuning).
    const char* force = getenv("QB200_HQ_KERNEL");
    // Measured crossover: below ~12 M elements the launch is one short wave and the CUDA-core kernel's smaller
    // set-up wins by about a microsecond.  Inside the one-call layer the crossover is 3 M elements: there the tcgen05
    // kernel and the GEMM behind it are launched with programmatic dependencies, which gains more than that
    // microsecond (M = 1024, K = N = 4096: 27.2 against 28.2 us per layer), while a GEMM launched that way behind
    // the CUDA-core kernel measured slower from 4 M elements on (29.5 us).
    const long long tc_from = qb_tl_dependent_quantiser ? kTcFromInLayer : 12ll * 1024 * 1024;
    const bool want_tc = force != nullptr ? (force[0] == 't') : ((long long)p.M * p.K >= tc_from);
    if (want_tc && hq_tc_eligible(p, block)) {
        qb_tl_quantiser_kernel = kQuantiserTc;
        switch (block) {
            case 64: return launch_hq_tc<64>(p, stream);
            case 128: return launch_hq_tc<128>(p, stream);
            default: return launch_hq_tc<256>(p, stream);
        }
    }
    if (force != nullptr && force[0] == 't') return QB200_ERR_UNSUPPORTED;
    qb_tl_quantiser_kernel = kQuantiserMma;
    switch (block) {
        case 64: return launch_hq_mma<64>(p, stream);
        case 128: return launch_hq_mma<128>(p, stream);
        default: return launch_hq_mma<256>(p, stream);
    }
}

// Producer-fused variants: the rows that are transformed and quantised are RMSNorm(x) * w, or SiLU(gate) * up, computed
// on the fly from the kernel's inputs (see hadamard_quant_mma_kernel).
static int run_producer_hq(RowParams& p, int block, int pro, cudaStream_t stream) {
    p.quantize = 1;
    p.had_scale = __bfloat162float(__float2bfloat16_rn((float)(1.0 / sqrt((double)block))));
    if (!vector_path_ok(p)) return QB200_ERR_UNSUPPORTED;
    if (pro == kProAddRmsNorm) {
        if (!aligned16(p.norm_w) || !aligned16(p.x2)) return QB200_ERR_UNSUPPORTED;
        switch (block) {
            case 64: return launch_hq_mma<64, kProAddRmsNorm>(p, stream);
            case 128: return launch_hq_mma<128, kProAddRmsNorm>(p, stream);
            default: return launch_hq_mma<256, kProAddRmsNorm>(p, stream);
        }
    }
    if (pro == kProRmsNorm) {
        if (!aligned16(p.norm_w)) return QB200_ERR_UNSUPPORTED;
        switch (block) {
            case 64: return launch_hq_mma<64, kProRmsNorm>(p, stream);
            case 128: return launch_hq_mma<128, kProRmsNorm>(p, stream);
            default: return launch_hq_mma<256, kProRmsNorm>(p, stream);
        }
    }
    if (!aligned16(p.x2)) return QB200_ERR_UNSUPPORTED;
    switch (block) {
        case 64: return launch_hq_mma<64, kProSiluMul>(p, stream);
        case 128: return launch_hq_mma<128, kProSiluMul>(p, stream);
        default: return launch_hq_mma<256, kProSiluMul>(p, stream);
    }
}

extern "C" int rmsnorm_hadamard_quantize_int4_cuda_bf16(void* x_int_packed_ptr, void* scale_ptr, void* x_int_row_sum_ptr,
                                                        const void* x_ptr, const void* norm_weight_ptr, float eps,
                                                        int group_size, int batch_size, int block, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (!x_int_packed_ptr || !scale_ptr || !x_ptr || !norm_weight_ptr || group_size == 0 || group_size % block != 0)
        return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.norm_w = static_cast<const __nv_bfloat16*>(norm_weight_ptr);
    p.norm_eps = eps;
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    p.q_packed = static_cast<uint8_t*>(x_int_packed_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.K = group_size;
    p.M = batch_size;
    return run_producer_hq(p, block, kProRmsNorm, stream);
}

extern "C" int producer_hadamard_quantize_cuda_bf16(void* codes_ptr, int int8_operand, void* scale_ptr, void* x_int_row_sum_ptr,
                                                    int producer, const void* x_ptr, const void* x2_ptr, void* sum_ptr,
                                                    const void* norm_weight_ptr, float eps, int group_size, int batch_size,
                                                    int block, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (producer != kProRmsNorm && producer != kProSiluMul && producer != kProAddRmsNorm) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (!codes_ptr || !scale_ptr || !x_ptr || group_size == 0 || group_size % block != 0) return QB200_ERR_INVALID_ARGUMENT;
    if (producer != kProSiluMul && !norm_weight_ptr) return QB200_ERR_INVALID_ARGUMENT;
    if (producer != kProRmsNorm && !x2_ptr) return QB200_ERR_INVALID_ARGUMENT;
    if (producer == kProAddRmsNorm && !sum_ptr) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.x2 = static_cast<const __nv_bfloat16*>(x2_ptr);
    p.x_out = producer == kProAddRmsNorm ? static_cast<__nv_bfloat16*>(sum_ptr) : nullptr;
    p.norm_w = static_cast<const __nv_bfloat16*>(norm_weight_ptr);
    p.norm_eps = eps;
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    if (int8_operand) p.q_a8 = static_cast<uint8_t*>(codes_ptr);
    else p.q_packed = static_cast<uint8_t*>(codes_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.K = group_size;
    p.M = batch_size;
    return run_producer_hq(p, block, producer, stream);
}

extern "C" int silu_mul_hadamard_quantize_int4_cuda_bf16(void* x_int_packed_ptr, void* scale_ptr, void* x_int_row_sum_ptr,
                                                         const void* gate_ptr, const void* up_ptr, int group_size,
                                                         int batch_size, int block, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (!x_int_packed_ptr || !scale_ptr || !gate_ptr || !up_ptr || group_size == 0 || group_size % block != 0)
        return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(gate_ptr);
    p.x2 = static_cast<const __nv_bfloat16*>(up_ptr);
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    p.q_packed = static_cast<uint8_t*>(x_int_packed_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.K = group_size;
    p.M = batch_size;
    return run_producer_hq(p, block, kProSiluMul, stream);
}

extern "C" int hadamard_quantize_a8_cuda_bf16(void* a8_ptr, void* scale_ptr, void* x_int_row_sum_ptr, const void* x_ptr,
                                              int group_size, int batch_size, int block, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (a8_ptr == nullptr || scale_ptr == nullptr || x_ptr == nullptr || group_size == 0) return QB200_ERR_INVALID_ARGUMENT;
    if (group_size % block != 0) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    p.q_a8 = static_cast<uint8_t*>(a8_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.K = group_size;
    p.M = batch_size;
    p.quantize = 1;
    p.had_scale = __bfloat162float(__float2bfloat16_rn((float)(1.0 / sqrt((double)block))));
    if (!hq_tc_eligible(p, block)) return QB200_ERR_UNSUPPORTED;
    p.let_dependents = qb_tl_in_layer;
    qb_tl_quantiser_kernel = kQuantiserTc;
    switch (block) {
        case 64: return launch_hq_tc<64>(p, stream);
        case 128: return launch_hq_tc<128>(p, stream);
        default: return launch_hq_tc<256>(p, stream);
    }
}

namespace qb {
int quantise_layer_operand(void* a8, void* scale, void* row_sum, const void* x, int K, int M, int block, cudaStream_t stream) {
    if (K < 0 || M < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 0 && block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (M == 0) return QB200_OK;
    if (a8 == nullptr || scale == nullptr || x == nullptr || K == 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 0 && K % block != 0) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x);
    p.scale_out = static_cast<__nv_bfloat16*>(scale);
    p.q_a8 = static_cast<uint8_t*>(a8);
    p.row_sum = static_cast<int32_t*>(row_sum);
    p.K = K;
    p.M = M;
    p.quantize = 1;
    p.let_dependents = qb_tl_in_layer;
    if (!vector_path_ok(p)) return QB200_ERR_UNSUPPORTED;
    if (block == 0) {
        qb_tl_quantiser_kernel = kQuantiserMma;
        return run_rows(p, 0, false, stream);
    }
    p.had_scale = __bfloat162float(__float2bfloat16_rn((float)(1.0 / sqrt((double)block))));
    const bool tc = hq_tc_eligible(p, block) && (long long)M * K >= kTcFromInLayer;
    qb_tl_quantiser_kernel = tc ? kQuantiserTc : kQuantiserMma;
    switch (block) {
        case 64: return tc ? launch_hq_tc<64>(p, stream) : launch_hq_mma<64>(p, stream);
        case 128: return tc ? launch_hq_tc<128>(p, stream) : launch_hq_mma<128>(p, stream);
        default: return tc ? launch_hq_tc<256>(p, stream) : launch_hq_mma<256>(p, stream);
    }
}
}  // namespace qb

extern "C" int hadamard_transform_cuda_bf16(void* out_ptr, const void* x_ptr, int group_size, int batch_size,
                                            int block, int weight_side, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (block != 64 && block != 128 && block != 256) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (out_ptr == nullptr || x_ptr == nullptr || group_size == 0 || group_size % block != 0)
        return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.x_out = static_cast<__nv_bfloat16*>(out_ptr);
    p.x_out_mode = 1;
    p.K = group_size;
    p.M = batch_size;
    p.quantize = 0;
    const float exact = (float)(1.0 / sqrt((double)block));  // fp32 rounding of block^-0.5
    p.had_scale = weight_side ? exact : __bfloat162float(__float2bfloat16_rn(exact));
    return run_rows(p, block, true, stream);
}

extern "C" int scale_quantize_int4_cuda_bf16(void* x_int_packed_ptr, void* scale_ptr, void* x_int_row_sum_ptr,
                                             const void* x_ptr, int group_size, int batch_size, int weight_block,
                                             int row_sum_add, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (weight_block != 0 && weight_block != 64 && weight_block != 128 && weight_block != 256) return QB200_ERR_UNSUPPORTED;
    if (batch_size == 0) return QB200_OK;
    if (!x_int_packed_ptr || !scale_ptr || !x_ptr || group_size == 0) return QB200_ERR_INVALID_ARGUMENT;
    if ((group_size & 1) || (weight_block != 0 && group_size % weight_block != 0)) return QB200_ERR_INVALID_ARGUMENT;
    RowParams p{};
    p.x = static_cast<const __nv_bfloat16*>(x_ptr);
    p.scale_out = static_cast<__nv_bfloat16*>(scale_ptr);
    p.q_packed = static_cast<uint8_t*>(x_int_packed_ptr);
    p.row_sum = static_cast<int32_t*>(x_int_row_sum_ptr);
    p.row_sum_add = row_sum_add;
    p.K = group_size;
    p.M = batch_size;
    p.quantize = 1;
    p.had_scale = weight_block != 0 ? (float)(1.0 / sqrt((double)weight_block)) : 1.f;  // weights carry the fp32 constant
    if (!vector_path_ok(p)) return QB200_ERR_UNSUPPORTED;
    return run_rows(p, weight_block, false, stream);
}

extern "C" int add_mul_vv_cuda_bf16(void* mat_d, const void* vec_a_add, const void* vec_a_mul, const void* vec_b_add,
                                    const void* vec_b_mul, const void* mat_c, int size_a, int size_b,
                                    cudaStream_t stream) {
    if (size_a < 0 || size_b < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (size_a == 0 || size_b == 0) return QB200_OK;
    if (!mat_d || !vec_a_add || !vec_a_mul || !vec_b_add || !vec_b_mul || !mat_c) return QB200_ERR_INVALID_ARGUMENT;
    auto* d = static_cast<__nv_bfloat16*>(mat_d);
    auto* aa = static_cast<const int32_t*>(vec_a_add);
    auto* am = static_cast<const __nv_bfloat16*>(vec_a_mul);
    auto* ba = static_cast<const int32_t*>(vec_b_add);
    auto* bm = static_cast<const __nv_bfloat16*>(vec_b_mul);
    auto* c = static_cast<const int32_t*>(mat_c);
    const long long total = (long long)size_a * size_b;
    const bool vec = (size_b % 8 == 0) && aligned16(d) && aligned16(c) && aligned16(ba) && aligned16(bm);
    const long long work = vec ? total / 8 : total;
    long long blocks = (work + 255) / 256;
    const long long cap = 148LL * 8 * 4;  // grid-stride beyond a few waves of the 148 SMs
    if (blocks > cap) blocks = cap;
    if (vec)
        add_mul_vv_vec8_kernel<<<(unsigned)blocks, 256, 0, stream>>>(d, aa, am, ba, bm, c, size_a, size_b);
    else
        add_mul_vv_scalar_kernel<<<(unsigned)blocks, 256, 0, stream>>>(d, aa, am, ba, bm, c, size_a, size_b);
    return launch_status();
}

extern "C" int rmsnorm_cuda_bf16(void* y, const void* x, const void* weight, float eps, int group_size, int batch_size, cudaStream_t stream) {
    if (group_size < 0 || batch_size < 0) return QB200_ERR_INVALID_ARGUMENT;
    if (group_size == 0 || batch_size == 0) return QB200_OK;
    if (!y || !x || !weight) return QB200_ERR_INVALID_ARGUMENT;
    if (group_size % 8 != 0 || !aligned16(y) || !aligned16(x) || !aligned16(weight)) return QB200_ERR_UNSUPPORTED;
    int blocks = (batch_size + 7) / 8;
    if (blocks > 148 * 16) blocks = 148 * 16;
    rmsnorm_kernel<<<blocks, 256, 0, stream>>>(static_cast<__nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(x),
                                               static_cast<const __nv_bfloat16*>(weight), batch_size, group_size, eps);
    return launch_status();
}

extern "C" int rope_inplace_cuda_bf16(void* x, const void* table, int table_is_bf16, int rows, int seq, int cols, int head_dim,
                                      long long ld, cudaStream_t stream) {
    if (rows < 0 || cols < 0 || seq <= 0 || head_dim <= 0 || ld < cols) return QB200_ERR_INVALID_ARGUMENT;
    if (rows == 0 || cols == 0) return QB200_OK;
    if (!x || !table) return QB200_ERR_INVALID_ARGUMENT;
    if (head_dim % 8 != 0 || cols % head_dim != 0 || ld % 8 != 0 || !aligned16(x) || !aligned16(table)) return QB200_ERR_UNSUPPORTED;
    const long long chunks = (long long)rows * (cols / 8);
    long long blocks = (chunks + 255) / 256;
    if (blocks > 148 * 64) blocks = 148 * 64;
    auto* p = static_cast<__nv_bfloat16*>(x);
    if (table_is_bf16)
        rope_inplace_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, stream>>>(p, static_cast<const __nv_bfloat16*>(table), chunks, cols / 8, seq, ld, head_dim);
    else
        rope_inplace_kernel<float><<<(unsigned)blocks, 256, 0, stream>>>(p, static_cast<const float*>(table), chunks, cols / 8, seq, ld, head_dim);
    return launch_status();
}

extern "C" int quest_b200_copy_block_to_peers_cuda(const void* src, void* const* dsts, int n_dst, int rows, int cols,
                                                   long long ld, cudaStream_t stream) {
    if (rows < 0 || cols < 0 || n_dst < 0 || n_dst > 7 || ld < cols) return QB200_ERR_INVALID_ARGUMENT;
    if (rows == 0 || cols == 0 || n_dst == 0) return QB200_OK;
    if (!src || !dsts) return QB200_ERR_INVALID_ARGUMENT;
    if (cols % 8 != 0 || ld % 8 != 0 || !aligned16(src)) return QB200_ERR_UNSUPPORTED;  // whole 16-byte pieces only
    CopyDsts d{};
    for (int i = 0; i < n_dst; ++i) {
        if (!dsts[i]) return QB200_ERR_INVALID_ARGUMENT;
        if (!aligned16(dsts[i])) return QB200_ERR_UNSUPPORTED;
        d.p[i] = dsts[i];
    }
    const int chunks = cols / 8;
    const long long total = (long long)rows * chunks;
    if (total > (1ll << 30)) return QB200_ERR_UNSUPPORTED;
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    copy_block_kernel<<<(unsigned)blocks, 256, 0, stream>>>(static_cast<const uint8_t*>(src), d, n_dst, rows, chunks, ld * 2);
    return launch_status();
}
