// The inner loop shared by the decode GEMVs whose warps multiply several row blocks with the same activations (gemv_rg.cu, gemv_moe.cu).
#pragma once
#include <type_traits>

#include "gemv_common.cuh"

namespace w4 {

struct RgKernel {
    const void* f;
    const char* name;
};
const RgKernel* rg_timeline_kernels();   // as rg_kernels of gemv_rg_kernel.cuh

constexpr int RG_WARPS = 8;
constexpr int RG_THREADS = RG_WARPS * 32;
constexpr int RG_XPAD = 32;            // bytes added to a token's row of x: 32 mod 128, conflict-free 8-byte reads of eight rows

// Ring slot of a warp: one k-block of its NR row blocks, then the scale words (groups of 32: two groups per k-block; groups of 128: with
// the group's second k-block).
__host__ __device__ constexpr int rg_weight_bytes(int nr) { return nr * TILE_WORDS * 4; }
__host__ __device__ constexpr int rg_slot_bytes(int group, int nr) { return rg_weight_bytes(nr) + nr * 32 * (group == 32 ? 2 : 1); }

// The warps' sums of a unit meet in shared memory as [warp along K][token][row], four floats of padding per token: what a lane holds -- rows g and
// g + 8 of two tokens -- goes to 32 banks, and consecutive rows come from 32.  As [row][token] every read of eight tokens' sums was an 8-way
// conflict, 1024 cycles a unit with eight warps along K: eight tokens of 7168 x 5120 7.6 -> 7.1 us, of 5120 x 17408 15.5 -> 14.6, of 2048 x 2048
// 3.0 -> 2.8; up to six tokens the same.
constexpr int RG_RED_PAD = 4;
__host__ __device__ constexpr int rg_red_pitch(int ur) { return ur * TILE_ROWS + RG_RED_PAD; }
__host__ __device__ constexpr int rg_red_bytes(int kw, int ur, int tokens) { return kw * tokens * rg_red_pitch(ur) * 4; }
template <int NR>
__device__ __forceinline__ void rg_store_sums(float* d, int pitch, const float (&tot)[NR][4], float m0, float m1) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        d[r * TILE_ROWS] = tot[r][0] * m0;
        d[r * TILE_ROWS + pitch] = tot[r][1] * m0;
        d[r * TILE_ROWS + 8] = tot[r][2] * m1;
        d[r * TILE_ROWS + pitch + 8] = tot[r][3] * m1;
    }
}

// A warp's ring and where its next slot comes from.  A slot is refilled as soon as it has been read, so one address serves both sides; a lane
// copies the weights that it reads itself.  Row blocks past the matrix are whatever lies behind it (the allocation is as much longer,
// TILE_READ_PAD), their sums are dropped; scales past it are those of the last row block.
template <int GROUP, int NR, int D>
struct RgStream {
    static constexpr uint32_t SLOT = rg_slot_bytes(GROUP, NR), SC = rg_weight_bytes(NR);
    const uint4* q;
    const uint32_t* s;
    size_t pitch;                      // uint4 between k-blocks
    int left;                          // k-blocks of the unit that are still to be requested
    uint32_t slot, first;              // this lane's 16 bytes of the slot in turn, of slot 0

    __device__ __forceinline__ void init(uint32_t ring, int lane) { slot = first = ring + (uint32_t)lane * 16u; }
    // `rb`: the warp's first row block, `nrb`: row blocks that it may take, both counted from `base` in a matrix of `nrb_all`; `kbs` k-blocks from kb0
    __device__ __forceinline__ void unit(const uint4* qt, const uint32_t* st, int base, int rb, int nrb, int nrb_all, int ng, int kb0, int kbs, int lane) {
        constexpr int SP = GROUP == 32 ? 4 : 2;                   // 16-byte pieces of scales per row block and slot
        pitch = (size_t)nrb_all * 32;
        q = qt + (size_t)kb0 * pitch + (size_t)(base + min(rb, nrb - 1)) * 32 + lane;
        s = st + (size_t)(base + min(rb + lane / SP % NR, nrb - 1)) * ng * 8 + (size_t)kb0 * TILE_K / GROUP * 8 + (lane % SP) * 4;
        left = kbs;
    }
    // requests the next k-block into the slot in turn; ODD: it is the second one of its group (groups of 128).  `next_unit` is called behind
    // a unit's last one.
    template <bool ODD, class Next>
    __device__ __forceinline__ void fetch(int lane, Next&& next_unit) {
        if (left > 0) {
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                cp_async_16(slot + (uint32_t)r * 512u, q + r * 32);
            }
            q += pitch;
            if (GROUP == 32 || ODD) {
                if (lane < (GROUP == 32 ? 4 : 2) * NR) {
                    cp_async_16(slot + SC, s);
                }
                s += GROUP == 32 ? 16 : 8;
            }
            if (--left == 0) {
                next_unit();
            }
        }
        cp_async_commit();
        if ((slot += SLOT) == first + D * SLOT) {
            slot = first;
        }
    }
};

// tot += the warp's NR row blocks times its tokens over nk k-blocks, in nibble units (rows g: 2^-24, rows g + 8: 2^-20).  `xa`: this
// lane's first activations; `next_unit` as in RgStream::fetch.
// The zero-point term of a group, -8 * sum(x), is the sum of MMAs whose A operand is the constant -8 in the nibbles' own two scalings: no
// pass over x, no table.  In groups of 32 it opens the chains of the row blocks as their C operand; in groups of 128, where it is complete
// only after the group's second k-block, it is added to their sums.
template <int GROUP, int NR, int D, class Next>
__device__ __forceinline__ void rg_multiply(float (&tot)[NR][4], uint32_t xa, int nk, RgStream<GROUP, NR, D>& ring, int lane, Next&& next_unit) {
    const uint32_t zA[4] = {0x80088008u, 0x80808080u, 0x80088008u, 0x80808080u};
    const uint32_t sl = rg_weight_bytes(NR) + (uint32_t)(lane >> 2) * 4u - (uint32_t)lane * 16u;   // from a lane's weights to its scales
    float acc[NR][4] = {};
    auto fold = [&](int r, uint32_t s2) {
        const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&s2));
        tot[r][0] = fmaf(acc[r][0], sf.x, tot[r][0]);
        tot[r][1] = fmaf(acc[r][1], sf.x, tot[r][1]);
        tot[r][2] = fmaf(acc[r][2], sf.y, tot[r][2]);
        tot[r][3] = fmaf(acc[r][3], sf.y, tot[r][3]);
    };
    if (GROUP == 32) {
        for (int i = 0; i < nk; ++i) {
            uint2 x[4];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                x[w] = lds64(xa + (uint32_t)w * 32u);
            }
            xa += TILE_K * 2;
            cp_async_wait_group<D - 1>();
            __syncwarp();                                 // the scale words are other lanes' copies
            uint4 wv[NR];
            uint32_t sc[NR][2];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                wv[r] = lds128(ring.slot + (uint32_t)r * 512u);
                sc[r][0] = lds32(ring.slot + sl + (uint32_t)r * 64u);
                sc[r][1] = lds32(ring.slot + sl + (uint32_t)r * 64u + 32u);
            }
            __syncwarp();
            ring.template fetch<true>(lane, next_unit);
            float z0[4], z1[4];
            mma16816_z(z0, zA, x[0].x, x[0].y);
            mma16816_z(z1, zA, x[2].x, x[2].y);
            mma16816(z0, zA, x[1].x, x[1].y);
            mma16816(z1, zA, x[3].x, x[3].y);
            const float4 c0 = make_float4(z0[0], z0[1], z0[2], z0[3]), c1 = make_float4(z1[0], z1[1], z1[2], z1[3]);
            uint32_t af[4];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                nibbles_as_subnormals(wv[r].x, af);
                mma16816_c(acc[r], af, x[0].x, x[0].y, c0);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                nibbles_as_subnormals(wv[r].y, af);
                mma16816(acc[r], af, x[1].x, x[1].y);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                fold(r, sc[r][0]);
                nibbles_as_subnormals(wv[r].z, af);
                mma16816_c(acc[r], af, x[2].x, x[2].y, c1);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                nibbles_as_subnormals(wv[r].w, af);
                mma16816(acc[r], af, x[3].x, x[3].y);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                fold(r, sc[r][1]);
            }
        }
    } else {
        for (int i = 0; i < nk; i += 2) {
            float z[4];
            uint32_t sc[NR];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint2 x[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    x[w] = lds64(xa + (uint32_t)w * 32u);
                }
                xa += TILE_K * 2;
                cp_async_wait_group<D - 1>();
                if (h == 1) {
                    __syncwarp();                         // the scale words are other lanes' copies
                }
                uint4 wv[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    wv[r] = lds128(ring.slot + (uint32_t)r * 512u);
                    if (h == 1) {
                        sc[r] = lds32(ring.slot + sl + (uint32_t)r * 32u);
                    }
                }
                __syncwarp();
                if (h == 0) {
                    ring.template fetch<false>(lane, next_unit);
                } else {
                    ring.template fetch<true>(lane, next_unit);
                }
                uint32_t af[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const bool open = h == 0 && w == 0;
                    if (open) {
                        mma16816_z(z, zA, x[w].x, x[w].y);
                    } else {
                        mma16816(z, zA, x[w].x, x[w].y);
                    }
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        nibbles_as_subnormals(w == 0 ? wv[r].x : w == 1 ? wv[r].y : w == 2 ? wv[r].z : wv[r].w, af);
                        if (open) {
                            mma16816_z(acc[r], af, x[w].x, x[w].y);
                        } else {
                            mma16816(acc[r], af, x[w].x, x[w].y);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[r][j] += z[j];
                }
                fold(r, sc[r]);
            }
        }
    }
}

// ---- one and two tokens: activations as signed digits
//
// mma.sync m16n8k32 on signed bytes takes the cycles of m16n8k16 on f16 for twice the channels, and two words of nibbles become its weight operand
// with six instructions instead of ten.  The activations of a warp's part of K are rounded to 23-bit integers in units that their largest one sets
// -- an f16 loses nothing until it is 2^9 times smaller than that one -- and cut into three signed digits of base 256, three columns of the MMA for a
// token.  Sums of a group are exact integers.  They start from a constant whose bits, read as f32, are 1.5 * 2^23, so that the sum plus that is an f32 without
// a conversion.
constexpr int RG_INT_ZERO = 0x4B400000;
constexpr float RG_F32_ZERO = 12582912.f;      // the same bits
__host__ __device__ constexpr int rg_digit_stride(int k) { return k + (k % 128 == 0 ? 64 : 128); }   // of a column: 64 mod 128, conflict-free 16-byte reads

__device__ __forceinline__ void mma16832(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16832_c(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const int (&c)[4]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
// Two words of a lane, 16 channels of two rows each -> the A operand of 32 channels, bytes in the order k, k + 2, k + 1, k + 3
__device__ __forceinline__ void nibbles_as_bytes(uint32_t w0, uint32_t w1, uint32_t (&a)[4]) {
    a[0] = w0 & 0x0f0f0f0fu;
    a[1] = (w0 >> 4) & 0x0f0f0f0fu;
    a[2] = w1 & 0x0f0f0f0fu;
    a[3] = (w1 >> 4) & 0x0f0f0f0fu;
}
// x in units that `zero`, 1.5 * 2^23 of them, sets, as the low 23 bits of the sum
__device__ __forceinline__ uint32_t add_f16(uint32_t x2, int half, float zero) {
    float r;
    if (half == 0) {
        asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tadd.rn.f32.f16 %0, l, %2;\n\t}" : "=f"(r) : "r"(x2), "f"(zero));
    } else {
        asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %1;\n\tadd.rn.f32.f16 %0, h, %2;\n\t}" : "=f"(r) : "r"(x2), "f"(zero));
    }
    return __float_as_uint(r);
}
// Four activations of neighbouring channels -> a word of each digit, in that byte order: d0 + 256 d1 + 65536 d2 units.  `zero`: 1.5 * 2^23 + 32896 units,
// `flip`: 0x40 in every byte, and 0x80 where the exponent of `zero` is odd.
__device__ __forceinline__ void split_digits(uint32_t x01, uint32_t x23, float zero, uint32_t flip, uint32_t (&d)[3]) {
    const uint32_t u0 = add_f16(x01, 0, zero), u1 = add_f16(x01, 1, zero), u2 = add_f16(x23, 0, zero), u3 = add_f16(x23, 1, zero);
    const uint32_t l02 = __byte_perm(u0, u2, 0x5140), l13 = __byte_perm(u1, u3, 0x5140);   // bytes 0, 0, 1, 1 of both
    d[0] = __byte_perm(l02, l13, 0x5410) ^ 0x80808080u;
    d[1] = __byte_perm(l02, l13, 0x7632) ^ 0x80808080u;
    const uint32_t v = __byte_perm(__byte_perm(u0, u2, 0x0062), __byte_perm(u1, u3, 0x0062), 0x5410) ^ flip;   // digit 2 of seven bits
    d[2] = v | ((v << 1) & 0x80808080u);
}
// packed maximum; a NaN stays
__device__ __forceinline__ uint32_t hmax2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.NaN.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Stages a warp's part of K (nk k-blocks from kb0 of m rows of `x`) as digits: columns [token][digit] of `stride` bytes at `dst`, the 16 bytes of
// a k-block that lane (g, t) multiplies together.  `raw`: 128 bytes of scratch per k-block and token.  The columns are shared by the `rws` warps
// that take this part of K; warp `rw` of them writes its share.  mul[token]: what a sum of digits is to be multiplied by.
__device__ __forceinline__ void rg_stage_digits(uint32_t dst, uint32_t stride, uint32_t raw, const uint16_t* x, int k, int m, int kb0, int nk, int rw, int rws, int lane,
                                                float (&mul)[RG_MAX_DIGIT_TOKENS]) {
    const int n = nk * 8;                                            // 16-byte pieces per token
    const bool two = m > 1;
    uint32_t mx[2] = {0u, 0u};
    x += kb0 * TILE_K;
    auto load = [&](auto loads) {                                    // (past the end: the last piece again)
        constexpr int U = decltype(loads)::value;
#pragma unroll 1
        for (int j0 = lane; j0 < n; j0 += two ? 16 * U : 32 * U) {
            uint4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                v[u] = ld_cg_128(x + (two && (u & 1) ? k : 0) + min(j0 + (two ? u >> 1 : u) * 32, n - 1) * 8);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                mx[u & 1] = hmax2(mx[u & 1], hmax2(hmax2(v[u].x & 0x7fff7fffu, v[u].y & 0x7fff7fffu), hmax2(v[u].z & 0x7fff7fffu, v[u].w & 0x7fff7fffu)));
                sts128(raw + (uint32_t)((two && (u & 1) ? n : 0) + min(j0 + (two ? u >> 1 : u) * 32, n - 1)) * 16u, v[u]);
            }
        }
    };
    if (m * n <= 128) {
        load(std::integral_constant<int, 4>());
    } else {
        load(std::integral_constant<int, 10>());
    }
    if (!two) {
        mx[0] = hmax2(mx[0], mx[1]);
    }
    __syncwarp();
#pragma unroll 1
    for (int tok = 0; tok < m; ++tok) {
        const uint32_t mt = tok ? mx[1] : mx[0], top = __reduce_max_sync(0xffffffffu, max(mt & 0xffffu, mt >> 16));
        const uint32_t e = top >> 10, ec = e > 0 ? e : 1;            // its exponent: |x| < 2^(ec - 14) = 2^21 units
        const float unit = __uint_as_float((127 - 35 + ec) << 23), zero = (RG_F32_ZERO + 32896.f) * unit;
        const uint32_t flip = (__float_as_uint(zero) & 0x800000u) ? 0xc0c0c0c0u : 0x40404040u;
        (tok ? mul[1] : mul[0]) = e == 31 ? __uint_as_float(0x7fc00000u) : unit;                     // infinities and NaN: NaN, as ever
        // piece c = channels 8 c .. + 7: words c / 2 % 4 of the lanes t = 2 (c % 2) and the next
        uint32_t d = dst + (uint32_t)(tok * 3) * stride + (uint32_t)(kb0 * TILE_K + (lane >> 3) * TILE_K + (lane & 1) * 32 + ((lane >> 1) & 3) * 4 + rw * (4 * TILE_K));
        uint32_t r = raw + (uint32_t)(tok * n + lane + 32 * rw) * 16u;
#pragma unroll 2
        for (int c = lane + 32 * rw; c < n; c += 32 * rws) {
            const uint4 v = lds128(r);
            uint32_t d0[3], d1[3];
            split_digits(v.x, v.y, zero, flip, d0);
            split_digits(v.z, v.w, zero, flip, d1);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                sts32(d + q * stride, d0[q]);
                sts32(d + q * stride + 16u, d1[q]);
            }
            d += (uint32_t)(rws * 4 * TILE_K);
            r += (uint32_t)rws * 512u;
        }
    }
}

// As rg_multiply, with digits: tot[.][0, 1] are rows g, [2, 3] rows g + 8 of columns 2t and 2t + 1, four to a token (three digits and one that is not
// looked at).  `xa`: this lane's 16 bytes of the first k-block in its column.  The zero point, -8 times the digits' sums, opens a group's chains
// (groups of 32) or is added to their sums.
template <int GROUP, int NR, int D, class Next>
__device__ __forceinline__ void rg_multiply_digits(float (&tot)[NR][4], uint32_t xa, int nk, RgStream<GROUP, NR, D>& ring, int lane, Next&& next_unit) {
    const uint32_t zA[4] = {0xf8f8f8f8u, 0xf8f8f8f8u, 0xf8f8f8f8u, 0xf8f8f8f8u};
    const int zero[4] = {RG_INT_ZERO, RG_INT_ZERO, RG_INT_ZERO, RG_INT_ZERO};
    const uint32_t sl = rg_weight_bytes(NR) + (uint32_t)(lane >> 2) * 4u - (uint32_t)lane * 16u;   // from a lane's weights to its scales
    int acc[NR][4] = {};
    auto fold = [&](int r, const float (&z)[4], uint32_t s2) {
        const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&s2));
        tot[r][0] = fmaf(__int_as_float(acc[r][0]) + z[0], sf.x, tot[r][0]);
        tot[r][1] = fmaf(__int_as_float(acc[r][1]) + z[1], sf.x, tot[r][1]);
        tot[r][2] = fmaf(__int_as_float(acc[r][2]) + z[2], sf.y, tot[r][2]);
        tot[r][3] = fmaf(__int_as_float(acc[r][3]) + z[3], sf.y, tot[r][3]);
    };
    if (GROUP == 32) {
        const float z[4] = {-RG_F32_ZERO, -RG_F32_ZERO, -RG_F32_ZERO, -RG_F32_ZERO};
#pragma unroll(NR == 1 ? 2 : 1)
        for (int i = 0; i < nk; ++i) {
            const uint4 x = lds128(xa);
            xa += TILE_K;
            int z0[4], z1[4];
            mma16832_c(z0, zA, x.x, x.y, zero);
            mma16832_c(z1, zA, x.z, x.w, zero);
            cp_async_wait_group<D - 1>();
            __syncwarp();                                            // the scale words are other lanes' copies
            uint4 wv[NR];
            uint32_t sc[NR][2], af[4];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                wv[r] = lds128(ring.slot + (uint32_t)r * 512u);
                sc[r][0] = lds32(ring.slot + sl + (uint32_t)r * 64u);
                sc[r][1] = lds32(ring.slot + sl + (uint32_t)r * 64u + 32u);
            }
            __syncwarp();
            ring.template fetch<true>(lane, next_unit);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                nibbles_as_bytes(wv[r].x, wv[r].y, af);
                mma16832_c(acc[r], af, x.x, x.y, z0);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                fold(r, z, sc[r][0]);
                nibbles_as_bytes(wv[r].z, wv[r].w, af);
                mma16832_c(acc[r], af, x.z, x.w, z1);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                fold(r, z, sc[r][1]);
            }
        }
    } else {
        for (int i = 0; i < nk; i += 2) {
            int z[4];
            uint32_t sc[NR], af[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 x = lds128(xa);
                xa += TILE_K;
                cp_async_wait_group<D - 1>();
                if (h == 1) {
                    __syncwarp();                                    // the scale words are other lanes' copies
                }
                uint4 wv[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    wv[r] = lds128(ring.slot + (uint32_t)r * 512u);
                    if (h == 1) {
                        sc[r] = lds32(ring.slot + sl + (uint32_t)r * 32u);
                    }
                }
                __syncwarp();
                if (h == 0) {
                    ring.template fetch<false>(lane, next_unit);
                    mma16832_c(z, zA, x.x, x.y, zero);
                } else {
                    ring.template fetch<true>(lane, next_unit);
                    mma16832(z, zA, x.x, x.y);
                }
                mma16832(z, zA, x.z, x.w);
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    nibbles_as_bytes(wv[r].x, wv[r].y, af);
                    if (h == 0) {
                        mma16832_c(acc[r], af, x.x, x.y, zero);
                    } else {
                        mma16832(acc[r], af, x.x, x.y);
                    }
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    nibbles_as_bytes(wv[r].z, wv[r].w, af);
                    mma16832(acc[r], af, x.z, x.w);
                }
            }
            float zf[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                zf[j] = __int_as_float(z[j]) - 2.f * RG_F32_ZERO;
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                fold(r, zf, sc[r]);
            }
        }
    }
}

}  // namespace w4
