// The inner loop shared by the decode GEMVs whose warps multiply several row blocks with the same activations (gemv_rg.cu, gemv_moe.cu).
#pragma once
#include "gemv_common.cuh"

namespace w4 {

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

}  // namespace w4
