// The Hadamard transform and the int4 quantisation of one warp-unit of a row (1024 elements), shared by the mma.sync
// quantiser and by the one-kernel layer for few rows.  Included inside no namespace.
#pragma once

#include "common.cuh"
#include "tcgen05.cuh"

namespace qb {

constexpr int kUnit = 1024;        // elements per warp-unit
constexpr float kFloorMagic = 12582912.0f;  // 1.5 * 2^23: adding it (round-down) leaves floor(y) in the low mantissa bits
constexpr int kFloorMagicBits = 0x4B400000;

// Element-wise clamp of a bf16 pair to [lo, hi] (both given as bf16 pairs).
__device__ __forceinline__ uint32_t clamp_bf16x2(uint32_t v, uint32_t lo, uint32_t hi) {
    uint32_t r;
    asm("{\n\t.reg .b32 t;\n\tmax.bf16x2 t, %1, %2;\n\tmin.bf16x2 %0, t, %3;\n\t}" : "=r"(r) : "r"(v), "r"(lo), "r"(hi));
    return r;
}

// Sum of the eight signed nibbles of w, times 16, accumulated into acc.
__device__ __forceinline__ int nibble_sum16(uint32_t w, int acc) {
    const uint32_t lo = (w << 4) & 0xF0F0F0F0u;
    const uint32_t hi = w & 0xF0F0F0F0u;
    acc = __dp4a((int)lo, 0x01010101, acc);
    acc = __dp4a((int)hi, 0x01010101, acc);
    return acc;
}

constexpr int kBlkPitch = 272;              // 256-byte block of 128 bf16 + 16 bytes of padding
constexpr int kStepIn = 8 * kBlkPitch;      // eight blocks per warp step
constexpr int kOutPitch = 80;               // 64 packed bytes per block + 16 bytes of padding
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool valid) {
    const int sz = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// Packed fp32 pairs (sm_100 executes add/sub/mul/fma on two floats per instruction).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpk2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { f32x2 r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 add2_rd(f32x2 a, f32x2 b) { f32x2 r; asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

// ---- B fragments: h * H16[k][o], MMA column n of tile nu is output o = 4*(n>>1) + 2*nu + (n&1) ----
__device__ __forceinline__ void hadamard16_fragments(float had_scale, int lane, uint32_t (&bfrag)[2][2]) {
    const int g = lane >> 2, tig = lane & 3;
    const uint32_t hb = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(had_scale));
#pragma unroll
    for (int nu = 0; nu < 2; ++nu) {
        const int o = 4 * (g >> 1) + 2 * nu + (g & 1);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int k0 = 2 * tig + 8 * half;
            const uint32_t lo = hb | ((__popc(k0 & o) & 1) ? 0x8000u : 0u);
            const uint32_t hi = hb | ((__popc((k0 + 1) & o) & 1) ? 0x8000u : 0u);
            bfrag[nu][half] = lo | (hi << 16);
        }
    }
}

// One unit, staged in shared memory as eight blocks of 128 bf16 with a pitch of kBlkPitch bytes: transform, round to bf16
// pairs v[2a + nu] (elements 16a + 4tig + 2nu (+1) of block g of the unit), add their squares to ssq2.
template <int HB>
__device__ __forceinline__ void transform_unit(uint32_t in_base, int lane, const uint32_t (&bfrag)[2][2], uint32_t (&v)[16], f32x2& ssq2) {
    const int g = lane >> 2;
                f32x2 f[8][2];  // f[a][h]: elements 16a + 4tig + 2h, +1 of block g, as packed float pairs
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        uint32_t a[4];
        ldmatrix_x4(in_base + (lane & 7) * kBlkPitch + (2 * t + ((lane >> 3) & 1)) * 32 + (lane >> 4) * 16, a);
#pragma unroll
        for (int nu = 0; nu < 2; ++nu) {
            float d[4];
            mma_bf16_16816(d, a, bfrag[nu][0], bfrag[nu][1]);
            f[2 * t][nu] = pk2(d[0], d[1]);
            f[2 * t + 1][nu] = pk2(d[2], d[3]);
        }
    }
    // remaining index bits 4.. of the block: butterflies over the row index a (in registers)
#pragma unroll
    for (int s = 1; s < 8 && s < HB / 16; s <<= 1) {
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            if ((a & s) == 0) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const f32x2 x0 = f[a][h], x1 = f[a + s][h];
                    f[a][h] = add2(x0, x1);
                    f[a + s][h] = sub2(x0, x1);
                }
            }
        }
    }
    if (HB == 256) {  // index bit 7 pairs neighbouring 128-element halves: lanes g and g ^ 1
        const float sgn = (g & 1) ? -1.f : 1.f;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float x0, x1;
                unpk2(f[a][h], x0, x1);
                const float p0 = __shfl_xor_sync(0xffffffffu, x0, 4);
                const float p1 = __shfl_xor_sync(0xffffffffu, x1, 4);
                f[a][h] = pk2(fmaf(x0, sgn, p0), fmaf(x1, sgn, p1));
            }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float x0, x1;
            unpk2(f[a][h], x0, x1);
            v[2 * a + h] = pack_bf16x2(x0, x1);
        }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const f32x2 xx = pk2(bf16lo_to_f32(v[i]), bf16hi_to_f32(v[i]));
        ssq2 = fma2(xx, xx, ssq2);
    }
}

// What the quantisation of a row needs of its scale.  Saturation is done on the bf16 pairs before the divide: x is clamped
// to [-8s, ~7.5s], both bounds exact or safely inside [7s, 8s), so floor(x/s) lands in [-8, 7] without integer min/max, and
// the code is simply the low nibble of the magic-number sum.
struct RowConstants {
    uint32_t lo2, hi2;
    f32x2 inv_s2;
};
__device__ __forceinline__ RowConstants row_constants(__nv_bfloat16 sb) {
    const float s_f = bf16_to_f32(sb);
    const float inv_s = __frcp_rn(s_f);
    const uint32_t lo1 = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(-8.f * s_f));
    const uint32_t hi1 = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(7.5f * s_f));
    return RowConstants{lo1 | (lo1 << 16), hi1 | (hi1 << 16), pk2(inv_s, inv_s)};
}

// Quantise and pack one transformed unit through the warp's staging area: the lane's 32 codes (elements 32 lane .. + 31 of
// the unit) as 16 packed bytes; adds sixteen times their sum to rs16.
__device__ __forceinline__ uint4 quantise_unit(const uint32_t (&v)[16], const RowConstants& rc, uint32_t out_base, int lane, int& rs16) {
    const int g = lane >> 2, tig = lane & 3;
    const uint32_t lo2 = rc.lo2, hi2 = rc.hi2;
    const f32x2 inv_s2 = rc.inv_s2, magic2 = pk2(kFloorMagic, kFloorMagic);
#pragma unroll
    for (int pr = 0; pr < 4; ++pr) {  // rows a = 2pr and 2pr + 1: eight codes -> one 32-bit word
        uint32_t ub[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t c = clamp_bf16x2(v[4 * pr + i], lo2, hi2);
            float y0, y1;
            unpk2(mul2(pk2(bf16lo_to_f32(c), bf16hi_to_f32(c)), inv_s2), y0, y1);
            // nudge towards +inf by |y| * 2^-13 (see floor_quotient), then floor through the magic-number sum
            const f32x2 fl = add2_rd(pk2(fmaf(fabsf(y0), 1.220703125e-4f, y0), fmaf(fabsf(y1), 1.220703125e-4f, y1)), magic2);
            float u0, u1;
            unpk2(fl, u0, u1);
            ub[2 * i] = __float_as_uint(u0);
            ub[2 * i + 1] = __float_as_uint(u1);
        }
        // ub[0..3] = row 2pr elements 0..3, ub[4..7] = row 2pr+1 elements 0..3; code = low nibble
        const uint32_t ev = __byte_perm(__byte_perm(ub[0], ub[2], 0x0040), __byte_perm(ub[4], ub[6], 0x0040), 0x5410);
        const uint32_t od = __byte_perm(__byte_perm(ub[1], ub[3], 0x0040), __byte_perm(ub[5], ub[7], 0x0040), 0x5410);
        const uint32_t word = (ev & 0x0F0F0F0Fu) | ((od << 4) & 0xF0F0F0F0u);
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(out_base + g * kOutPitch + pr * 16 + tig * 4), "r"(word) : "memory");
    }
    __syncwarp();
    uint4 t4;  // lane reads rows (2c, 2c+1) of block lane>>2, c = lane&3: one word per source thread tig
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(t4.x), "=r"(t4.y), "=r"(t4.z), "=r"(t4.w) : "r"(out_base + (lane >> 2) * kOutPitch + (lane & 3) * 16));
    __syncwarp();  // the staging area is rewritten for the next row
    uint4 w;   // low halves are row 2c (bytes 2tig, 2tig+1), high halves row 2c+1
    w.x = __byte_perm(t4.x, t4.y, 0x5410);
    w.y = __byte_perm(t4.z, t4.w, 0x5410);
    w.z = __byte_perm(t4.x, t4.y, 0x7632);
    w.w = __byte_perm(t4.z, t4.w, 0x7632);
    rs16 = nibble_sum16(w.x, rs16);
    rs16 = nibble_sum16(w.y, rs16);
    rs16 = nibble_sum16(w.z, rs16);
    rs16 = nibble_sum16(w.w, rs16);
    return w;
}

}  // namespace qb
