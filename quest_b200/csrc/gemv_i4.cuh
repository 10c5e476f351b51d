// int4 x int4 GEMM for very few activation rows (M <= 16, decode-like shapes) on the CUDA cores.  Included by
// gemm_i4.cu inside namespace qb.
//
// With so few rows the layer is a stream over the packed weights (N * K / 2 bytes, read once) and the tensor-core
// kernels spend most of their time on set-up and on walking K serially.  Here every warp owns C weight rows (output
// columns) at a time and splits K over its lanes: a lane loads 16 packed bytes (32 codes) per weight row and step,
// unpacks them to two int8x4 groups with the same "times sixteen" trick as the tensor-core path
// ((w << 4) & 0xF0F0F0F0 and w & 0xF0F0F0F0: sixteen times the low / high nibble codes, no sign extension needed),
// and multiplies them with dp4a against the activation rows, which the block has staged - packed - in shared memory.
// Both operands carry the factor 16, so the sums carry exactly 256 and are shifted back after the warp reduction
// (redux.sync); the fused epilogue is the same exact expression as everywhere else.
//
// Replaces, for these shapes, gemm-quest/quest/matmul_kernel.cu:8-63 and fused_matmul_dequantize_kernel.cu:4-57.
#pragma once

namespace gemv {
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxStageBytes = 112 * 1024;  // packed activations of all rows must fit in shared memory
}  // namespace gemv

__device__ __forceinline__ int redux_add(int v) {
    int r;
    asm volatile("redux.sync.add.s32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
    return r;
}

// MR: activation rows held (M <= MR; missing rows are zero).  C: weight rows per warp step (MR * C <= 32).
template <int C>
__device__ __forceinline__ void gemv_load_weights(uint4 (&w)[C], const uint8_t* __restrict__ B, int n0, int ch, int chunks, int N) {
    const size_t row_bytes = (size_t)chunks * 16;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const bool in = ch < chunks && n0 + c < N;
        w[c] = in ? ld_stream16(B + (size_t)(n0 + c) * row_bytes + (size_t)ch * 16) : make_uint4(0, 0, 0, 0);
    }
}

// The product of the activations staged in shared memory ([MR][K / 32] chunks of 16 packed bytes) with this warp's weight
// rows, and the epilogue.  wcur holds the first weights of the warp's first group.
template <int MR, int C, bool FUSED>
__device__ __forceinline__ void gemv_main(const uint4* gemv_sA, const uint8_t* __restrict__ B, const EpilogueParams& ep,
                                          const int32_t* a_add, const __nv_bfloat16* a_mul, uint4 (&wcur)[C], int M, int N, int K) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunks = K >> 5, groups = (N + C - 1) / C, steps = (chunks + 31) >> 5;
    int group = blockIdx.x * gemv::kWarps + warp;
    for (; group < groups; group += gridDim.x * gemv::kWarps) {
        const int n0 = group * C;
        int acc[MR][C];
#pragma unroll
        for (int m = 0; m < MR; ++m)
#pragma unroll
            for (int c = 0; c < C; ++c) acc[m][c] = 0;
        for (int j = 0; j < steps; ++j) {
            const int ch = lane + 32 * j;
            uint4 wnext[C];
            if (j + 1 < steps) {
                gemv_load_weights(wnext, B, n0, ch + 32, chunks, N);
            } else {  // the first step of this warp's next group
                const int g2 = group + gridDim.x * gemv::kWarps;
                gemv_load_weights(wnext, B, g2 * C, g2 < groups ? lane : chunks, chunks, N);
            }
            uint32_t wl[C][4], wh[C][4];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t w4[4] = {wcur[c].x, wcur[c].y, wcur[c].z, wcur[c].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    wl[c][i] = (w4[i] << 4) & 0xF0F0F0F0u;
                    wh[c][i] = w4[i] & 0xF0F0F0F0u;
                }
            }
            if (ch < chunks) {
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    const uint4 a = gemv_sA[m * chunks + ch];
                    const uint32_t a4[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int al = (int)((a4[i] << 4) & 0xF0F0F0F0u), ah = (int)(a4[i] & 0xF0F0F0F0u);
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            acc[m][c] = __dp4a(al, (int)wl[c][i], acc[m][c]);
                            acc[m][c] = __dp4a(ah, (int)wh[c][i], acc[m][c]);
                        }
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) wcur[c] = wnext[c];
        }
        // warp totals; lane o keeps output (row o / C, column o % C)
        int mine = 0;
#pragma unroll
        for (int m = 0; m < MR; ++m)
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int t = redux_add(acc[m][c]);
                if (lane == m * C + c) mine = t;
            }
        const int m = lane / C, n = n0 + lane % C;
        if (lane < MR * C && m < M && n < N) {
            const int v = mine >> 8;  // exact: both operands carried the factor 16
            if (FUSED) {
                const float f = (float)(2 * v + a_add[m] + ep.b_add[n]) * (0.5f * bf16_to_f32(a_mul[m]) * bf16_to_f32(ep.b_mul[n]));
                __nv_bfloat16 y = __float2bfloat16_rn(f);
                if (ep.bias != nullptr) y = __float2bfloat16_rn(bf16_to_f32(y) + bf16_to_f32(ep.bias[n]));
                static_cast<__nv_bfloat16*>(ep.out)[(size_t)m * ep.ld + n] = y;
            } else {
                static_cast<int32_t*>(ep.out)[(size_t)m * ep.ld + n] = v;
            }
        }
    }
}

template <int MR, int C, bool FUSED>
__global__ void __launch_bounds__(gemv::kThreads)
gemv_i4_kernel(const uint8_t* __restrict__ A, const uint8_t* __restrict__ B, const EpilogueParams ep, const int M,
               const int N, const int K) {
    extern __shared__ uint4 gemv_sA[];  // [MR][K / 32] chunks of 16 packed bytes
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunks = K >> 5;          // 32 codes = 16 bytes per chunk
    const size_t row_bytes = (size_t)(K >> 1);
    // The first weights are requested before the activations are staged: both latencies overlap.
    const int group = blockIdx.x * gemv::kWarps + warp;
    uint4 wcur[C];
    gemv_load_weights(wcur, B, group * C, group < (N + C - 1) / C ? lane : chunks, chunks, N);
    // Launched with a programmatic dependency on the kernel that quantises the activations (fused layer call), this
    // grid starts while that kernel still runs: everything up to here touches only the weights.  Now wait for it.
    wait_for_preceding_grid();
    for (int i = threadIdx.x; i < MR * chunks; i += gemv::kThreads) {
        const int r = i / chunks, ch = i - r * chunks;
        gemv_sA[i] = r < M ? *reinterpret_cast<const uint4*>(A + (size_t)r * row_bytes + (size_t)ch * 16) : make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    gemv_main<MR, C, FUSED>(gemv_sA, B, ep, ep.a_add, ep.a_mul, wcur, M, N, K);
}

// The whole layer in one kernel, for so few rows that every block can transform and quantise them itself: the block's
// eight warps hold one row part each (UNITS units of 1024 elements; W parts per row, dealt out and summed exactly as
// hadamard_quant_mma_kernel does, so the codes and scales are the same bits), the codes stay in shared memory, and a launch,
// its tail and the workspaces fall away.  The first weights are on their way meanwhile.  What bounds it is latency: about a
// microsecond for the rows to arrive and as much for the quantisation, behind the launch.
template <int MR, int C, int HB, int UNITS>
__global__ void __launch_bounds__(gemv::kThreads, 2)
gemv_layer_kernel(const __nv_bfloat16* __restrict__ x, const uint8_t* __restrict__ B, const EpilogueParams ep, const int M,
                  const int N, const int K, const int W, const float had_scale) {
    extern __shared__ uint4 gemv_sA[];  // the codes, then one staging area per warp
    __shared__ float part_ssq[gemv::kWarps];
    __shared__ int part_rs[gemv::kWarps];
    __shared__ int row_add[MR];
    __shared__ __nv_bfloat16 row_mul[MR];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chunks = K >> 5;
    const int group = blockIdx.x * gemv::kWarps + warp;
    uint4 wcur[C];
    gemv_load_weights(wcur, B, group * C, group < (N + C - 1) / C ? lane : chunks, chunks, N);

    const int row = warp / W, wig = warp - row * W;  // this warp's row part
    const bool busy = row < M;
    const uint32_t stage = smem_u32(gemv_sA) + (uint32_t)(MR * chunks * 16 + warp * UNITS * kStepIn);
    if (busy) {
        const __nv_bfloat16* xr = x + (size_t)row * K;
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = j * 32 + lane;  // 16-byte chunk within the unit
                const int e = (u * W + wig) * kUnit + c * 8;
                const bool valid = e < K;
                cp_async16_zfill(stage + u * kStepIn + (c >> 4) * kBlkPitch + (c & 15) * 16, valid ? (const void*)(xr + e) : (const void*)xr, valid);
            }
        }
    }
    for (int i = M * chunks + threadIdx.x; i < MR * chunks; i += gemv::kThreads) gemv_sA[i] = make_uint4(0, 0, 0, 0);
    uint32_t bfrag[2][2];
    hadamard16_fragments(had_scale, lane, bfrag);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    uint32_t v[UNITS][16];
    if (busy) {  // warp-uniform
        f32x2 ssq2 = 0ull;
#pragma unroll
        for (int u = 0; u < UNITS; ++u) transform_unit<HB>(stage + u * kStepIn, lane, bfrag, v[u], ssq2);
        float s0, s1;
        unpk2(ssq2, s0, s1);
        float ssq = s0 + s1;
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, m);
        if (lane == 0) part_ssq[warp] = ssq;
    }
    __syncthreads();
    if (busy) {
        double tot = 0.0;
        for (int i = 0; i < W; ++i) tot += (double)part_ssq[row * W + i];
        const __nv_bfloat16 sb = __float2bfloat16_rn(quest_scale_from_mean_square(__fdiv_rn((float)tot, (float)K)));
        const RowConstants rc = row_constants(sb);
        if (wig == 0 && lane == 0) row_mul[row] = sb;
        int rs16 = 0;
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const uint4 w = quantise_unit(v[u], rc, stage + u * kStepIn, lane, rs16);
            const int e0 = (u * W + wig) * kUnit + lane * 32;
            if (e0 < K) gemv_sA[row * chunks + (e0 >> 5)] = w;
        }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) rs16 += __shfl_xor_sync(0xffffffffu, rs16, m);
        if (lane == 0) part_rs[warp] = rs16;
    }
    __syncthreads();
    if (threadIdx.x < M) {
        int t = 0;
        for (int i = 0; i < W; ++i) t += part_rs[threadIdx.x * W + i];
        row_add[threadIdx.x] = t >> 4;  // exact: every term is a multiple of 16
    }
    __syncthreads();
    gemv_main<MR, C, true>(gemv_sA, B, ep, row_add, row_mul, wcur, M, N, K);
}

// dp4a runs at half the CUDA-core rate, so the kernel is compute-bound from a few rows on: it is used while the whole
// product stays below 2^28 multiply-adds (~7 us of dp4a), beyond that the tensor-core kernels win (measured).
static bool gemv_eligible(int M, int K, int N, int n_peer) {
    if (M < 1 || M > 16 || n_peer != 0) return false;
    if ((long long)M * N * K > (1ll << 28)) return false;
    const int mr = M <= 1 ? 1 : (M <= 2 ? 2 : (M <= 4 ? 4 : (M <= 8 ? 8 : 16)));
    return (size_t)mr * (size_t)(K / 2) <= (size_t)gemv::kMaxStageBytes;
}

template <int MR, int C, bool FUSED>
static int launch_gemv(const EpilogueParams& ep, const void* a, const void* b, int M, int K, int N, int sms, int dev,
                       cudaStream_t stream) {
    static bool attr_set[64] = {false};
    auto kernel = gemv_i4_kernel<MR, C, FUSED>;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gemv::kMaxStageBytes) != cudaSuccess) {
            cudaGetLastError();
            return QB200_ERR_CUDA;
        }
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const size_t smem = (size_t)MR * (size_t)(K / 2);
    const int groups = (N + C - 1) / C;
    int grid = (groups + gemv::kWarps - 1) / gemv::kWarps;
    const int per_sm = smem > 100 * 1024 ? 1 : (smem > 48 * 1024 ? 2 : 4);
    if (grid > sms * per_sm) grid = sms * per_sm;
    if (launch_kernel(kernel, grid, gemv::kThreads, smem, stream, static_cast<const uint8_t*>(a), static_cast<const uint8_t*>(b), ep, M, N, K) != cudaSuccess) {
        cudaGetLastError();
        return QB200_ERR_CUDA;
    }
    return launch_status();
}

template <bool FUSED>
static int run_gemv(const EpilogueParams& ep, const void* a, const void* b, int M, int K, int N, int sms, int dev,
                    cudaStream_t stream) {
    if (M <= 1) return launch_gemv<1, 4, FUSED>(ep, a, b, M, K, N, sms, dev, stream);
    if (M <= 2) return launch_gemv<2, 4, FUSED>(ep, a, b, M, K, N, sms, dev, stream);
    if (M <= 4) return launch_gemv<4, 4, FUSED>(ep, a, b, M, K, N, sms, dev, stream);
    if (M <= 8) return launch_gemv<8, 4, FUSED>(ep, a, b, M, K, N, sms, dev, stream);
    return launch_gemv<16, 2, FUSED>(ep, a, b, M, K, N, sms, dev, stream);
}

// Rows that one block can quantise with a warp per row part (W parts of `per` units, as hadamard_quant_mma_kernel deals
// them out), behind the Hadamard transform, while two blocks per SM hold all weight rows at once.  Per layer, weights from
// HBM, two kernels / one: M 1 K 4096 N 4096 7.7 / 6.6 us, M 4 8.2 / 8.2, M 1 K 2048 N 5632 6.1 / 5.6, M 2 K 8192 N 3584
// 10.7 / 10.3.  Near the end of the range it takes up to a microsecond more (M 2 K 4096 N 8192 8.7 / 9.5) and saves the
// caller a launch and an allocation (a call 16.5 / 11.2).  In a second round of blocks most SMs would idle, and every block
// repeats the rows (M 1 K 4096 N 11008 9.2 / 11.5, K 8192 N 10240 12.9 / 17.0; with three blocks per SM 10.2 and 14.2).
// Beyond 100 M multiply-adds the plain kernel's four blocks per SM stream the weights faster.
constexpr int kLayerBlocksPerSm = 2, kLayerC = 4;
static int gemv_layer_parts(int M, int K, int N, int block, int sms, int* per_out) {
    if (M < 1 || M > 4 || (block != 64 && block != 128 && block != 256) || K % block != 0) return 0;
    if (!gemv_eligible(M, K, N, 0) || (long long)M * N * K > 100000000ll) return 0;
    if ((long long)N > (long long)kLayerC * gemv::kWarps * kLayerBlocksPerSm * sms) return 0;
    const int units = (K + kUnit - 1) / kUnit;
    const int per = units >= 2 ? 2 : 1;
    const int W = (units + per - 1) / per;
    *per_out = per;
    return M * W <= gemv::kWarps ? W : 0;
}

template <int MR, int HB, int UNITS>
static int launch_gemv_layer(const EpilogueParams& ep, const void* x, const void* b, int M, int K, int N, int W, int sms, int dev,
                             cudaStream_t stream) {
    constexpr int C = kLayerC;
    static bool attr_set[64] = {false};
    auto kernel = gemv_layer_kernel<MR, C, HB, UNITS>;
    const size_t smem = (size_t)MR * (size_t)(K / 2) + (size_t)gemv::kWarps * UNITS * kStepIn;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) {
            cudaGetLastError();
            return QB200_ERR_CUDA;
        }
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const int grid = ((N + C - 1) / C + gemv::kWarps - 1) / gemv::kWarps;  // all resident, see gemv_layer_parts
    const float had_scale = __bfloat162float(__float2bfloat16_rn((float)(1.0 / sqrt((double)HB))));
    kernel<<<grid, gemv::kThreads, smem, stream>>>(static_cast<const __nv_bfloat16*>(x), static_cast<const uint8_t*>(b), ep, M, N, K, W, had_scale);
    return launch_status();
}

template <int MR, int HB>
static int launch_gemv_layer_units(const EpilogueParams& ep, const void* x, const void* b, int M, int K, int N, int sms, int dev,
                                   cudaStream_t stream) {
    int per = 0;
    const int W = gemv_layer_parts(M, K, N, HB, sms, &per);
    if (W == 0) return QB200_ERR_UNSUPPORTED;
    if (per == 1) return launch_gemv_layer<MR, HB, 1>(ep, x, b, M, K, N, W, sms, dev, stream);
    return launch_gemv_layer<MR, HB, 2>(ep, x, b, M, K, N, W, sms, dev, stream);
}

static int run_gemv_layer(const EpilogueParams& ep, const void* x, const void* b, int M, int K, int N, int block, int sms, int dev,
                          cudaStream_t stream) {
#define QB_GEMV_LAYER(HB)                                                                       \
    (M <= 1 ? launch_gemv_layer_units<1, HB>(ep, x, b, M, K, N, sms, dev, stream)               \
            : M <= 2 ? launch_gemv_layer_units<2, HB>(ep, x, b, M, K, N, sms, dev, stream)      \
                     : launch_gemv_layer_units<4, HB>(ep, x, b, M, K, N, sms, dev, stream))
    switch (block) {
        case 64: return QB_GEMV_LAYER(64);
        case 128: return QB_GEMV_LAYER(128);
        case 256: return QB_GEMV_LAYER(256);
        default: return QB200_ERR_UNSUPPORTED;
    }
#undef QB_GEMV_LAYER
}
