// Prefill W4A16 GEMM on the 5th-generation tensor cores:  y[m][n] = sum_k x[m][k] * f16((q[n][k]-8)*s[n][k/g]).
//
// Takes the place of the reference's prefill GEMMs (vendored Marlin instantiations launched from
// crates/backend-gpu/src/rawcuda/w4a16_dec/kernels/marlin.rs:94-213, and the hand-written
// crates/backend-gpu/src/rawcuda/assets/moe.cu:1139-1587 / gptq4.cu:984-1147), which are mma.sync kernels.
// Like them it multiplies the dequantised weight ROUNDED ONCE TO F16 (hmul2 of the exact integer and
// the f16 scale; the reference's own model of this is crates/server/src/probes/w4a16/gpu/bench.rs:240)
// and accumulates in f32.
//
// One CTA computes a tile of 128 or 256 tokens x 256 weight rows (128..224 where that fills SMs which 256 leaves idle).  The
// issuing warps stay converged with one elected lane (4096 tokens, four linears of a 27B-class layer: 2390 -> 2338 us).
//   warp 0      producer: TMA-loads the f16 activation tile (128 x 64, 128B swizzle) and bulk-copies the
//               raw int4 tiles (16 x 512 B of the T64 layout) of each 64-wide k-block into a 6-stage ring
//   warps 2-17  expand int4 -> f16 into a 2-stage ring of K-major 128B-swizzled B operands (a lane's word holds 4
//               consecutive k of two weight rows: 8-byte pieces, half a swizzled chunk), then signal the MMA warp
//   warp 1      issues 4 x tcgen05.mma (M128, N = weight rows of the tile, K16, f16 x f16 -> f32 in TMEM) per k-block
//               and 128-token block and commits the stage back to the producer
//   warps 2-17  epilogue: tcgen05.ld the f32 accumulators (each warp its TMEM lane quadrant, every fourth
//               32-column chunk), convert, store y
// Every mbarrier wait is bounded: on expiry the kernel records a status code, all roles fall through to
// the common exit, TMEM is released, and the host reports an error instead of hanging.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <string>

#include "../../include/w4a16_b200.h"
#include "dec.h"
#include "gemm_common.cuh"
#include "ptx.cuh"

namespace w4 {

namespace {

constexpr int BM = 128;           // tokens per tile (UMMA M)
constexpr int BN = 256;           // weight rows per tile (UMMA N)
constexpr int BK = TILE_K;        // 64 k per stage = one 128-byte swizzle row of f16
constexpr int A_BYTES = BM * BK * 2;          // 16 KB per 128-token block
constexpr int RAW_BYTES = BN * BK / 2;        // 8 KB
constexpr int B_BYTES = BN * BK * 2;          // 32 KB
constexpr int NUM_DQ_WARPS = 16;   // one 16-row block of the tile each
constexpr int NUM_THREADS = (2 + NUM_DQ_WARPS) * 32;
// MT = 128-token blocks per CTA tile (1 or 2).  With MT = 2 one expanded weight stage feeds two MMAs groups
// (two TMEM accumulators), halving the expand work and the shared-memory traffic per flop.
template <int MT> struct Cfg {
    static constexpr int NT = MT == 1 ? 6 : 4;   // TMA ring: activation blocks + raw int4 tile per stage
    static constexpr int NB = 2;                 // ring of expanded f16 weight tiles (3 with a shallower TMA ring measured slower)
    static constexpr int A_STAGE = MT * A_BYTES;
    static constexpr int TMEM_COLS = 256 * MT;
    static constexpr int SMEM = NT * (A_STAGE + RAW_BYTES) + NB * B_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
};
constexpr int GROUP_M = 8;        // m-tiles per rasterisation group (L2 reuse of the weight tiles)

struct GemmArgs {
    const uint32_t* qt;
    const uint32_t* st;  // scale pairs
    void* out;
    int m, n, k;
    int out_f16;
    int m_tiles, n_tiles;
    int bn;          // weight rows per tile = MMA N: a multiple of 32 up to BN (BN when grouped)
    int nrb_w;       // 16-row blocks of the resident weight matrix (= n/16; experts stacked along n when grouped)
    // grouped (MoE) mode: m-tiles come from a device table, one expert's weights per tile
    int grouped;
    const int* tile_expert;
    const int* tile_row0;
    const int* tile_rows;
    const int* num_tiles;
    int expert0;          // first expert held by this decoder
    const float* row_w;   // optional per-row factor applied in the epilogue (routing weight)
    float out_mul;        // power of two applied to every sum (undoes the shift of bf16 scales; normally 1)
    int glu;              // 1: weight rows are interleaved gate / up 16-row blocks; the epilogue stores
                          // f16(silu(f16 gate) * f16 up), n/2 values per row
    // split-K: the first `n_whole` tiles (in launch order) are one CTA each; every later tile is `ksplit` CTAs, each
    // multiplying k-blocks [nkb*s/ksplit, nkb*(s+1)/ksplit).  Their f32 partial tiles go to `part`, and the last
    // splits of a tile add a slice each, in split order (ticket per tile, left at zero), convert and store.  Used for the
    // tiles of an incomplete last wave, and for all tiles where there are too few of them and the weight-row form
    // (gemm_ts.cu) is not estimated faster.
    int n_whole;
    int ksplit;
    float* part;          // [split tiles][ksplit][BM*MT][BN] f32
    unsigned* counters;   // [split tiles]
    int* status;  // 0 = ok; otherwise code<<16 | detail of the first wait that expired
    long long* dbg;  // optional timeline buffer (diagnostic), CTA 0 only
    int tma_store;   // 1: whole dense tiles leave through shared memory and TMA stores (tmap_y)
};

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

template <int GROUP, int MT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_w4a16_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y,
                     const GemmArgs a) {
    constexpr int NT = Cfg<MT>::NT;
    constexpr int NB = Cfg<MT>::NB;
    constexpr int A_STAGE = Cfg<MT>::A_STAGE;
    constexpr int TMEM_COLS = Cfg<MT>::TMEM_COLS;
    constexpr int BMT = BM * MT;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ int s_last;

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // known to be warp-uniform
    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
    // [A ring NT x MT*16K][B ring NB x 32K][raw ring NT x 8K][barriers]; A and B bases are 1024-byte aligned
    auto a_addr = [&](int s) { return base + (uint32_t)s * A_STAGE; };
    auto b_addr = [&](int s) { return base + (uint32_t)(NT * A_STAGE) + (uint32_t)s * B_BYTES; };
    auto raw_addr = [&](int s) { return base + (uint32_t)(NT * A_STAGE + NB * B_BYTES) + (uint32_t)s * RAW_BYTES; };
    const uint32_t bars = base + NT * (A_STAGE + RAW_BYTES) + NB * B_BYTES;
    auto full_bar = [&](int s) { return bars + 8u * s; };               // TMA landed (A + raw)
    auto empty_bar = [&](int s) { return bars + 8u * (NT + s); };       // MMAs that read A[s] retired
    auto bready_bar = [&](int s) { return bars + 8u * (2 * NT + s); };  // B[s] expanded
    auto bfree_bar = [&](int s) { return bars + 8u * (2 * NT + NB + s); };  // MMAs that read B[s] retired
    const uint32_t accum_bar = bars + 8u * (2 * NT + 2 * NB);

    // tile of this CTA (groups of GROUP_M m-tiles walk the n-tiles together)
    int m0, n0, rb0, rows_valid;
    // whole tiles first, then the split ones: their CTAs run last and fill the wave the whole tiles leave incomplete
    const bool is_split = (int)blockIdx.x >= a.n_whole && a.ksplit > 1;
    const int ks = is_split ? a.ksplit : 1;
    const int sidx = is_split ? ((int)blockIdx.x - a.n_whole) / ks : 0;     // index among the split tiles
    const int split = is_split ? ((int)blockIdx.x - a.n_whole) % ks : 0;
    const int tile_id = is_split ? a.n_whole + sidx : (int)blockIdx.x;
    if (a.grouped) {
        // Consecutive CTAs walk the n-tiles of one m-tile, then the expert's next m-tile: a tile's token rows are read while they
        // are in L2 and so are the expert's weights.  (The other way round each n-tile read all sorted rows again, 134 MB at 4096
        // tokens x 8 experts x 2048 channels: 537 us per layer, 505 this way.)
        const int mt = tile_id / a.n_tiles, n_tile = tile_id - mt * a.n_tiles;
        if (mt >= *a.num_tiles) {
            return;  // the table is sized for the worst case
        }
        m0 = a.tile_row0[mt];
        rows_valid = a.tile_rows[mt];
        n0 = n_tile * a.bn;
        rb0 = ((a.tile_expert[mt] - a.expert0) * a.n + n0) / TILE_ROWS;
    } else {
        // groups of GROUP_M m-tiles walk the n-tiles together
        const int tile = tile_id;
        const int per_group = GROUP_M * a.n_tiles;
        const int grp = tile / per_group;
        const int first_m = grp * GROUP_M;
        const int gsz = min(GROUP_M, a.m_tiles - first_m);
        const int rem = tile - grp * per_group;
        m0 = (first_m + rem % gsz) * BMT;
        n0 = (rem / gsz) * a.bn;
        rb0 = n0 / TILE_ROWS;
        rows_valid = min(BMT, a.m - m0);
    }
    const int nkb_all = a.k / BK;
    const int kb0 = (int)((long long)nkb_all * split / ks);                 // this split's k-blocks: [kb0, kb0 + nkb)
    const int nkb = (int)((long long)nkb_all * (split + 1) / ks) - kb0;
    const int nrbv = min(a.bn, a.n - n0) / TILE_ROWS;  // valid 16-row blocks in this tile
    // 128-token blocks of this tile that hold rows: an empty second block is neither fetched nor multiplied
    const int mt_live = (MT == 2 && rows_valid <= BM) ? 1 : MT;

    const bool stamp = a.dbg != nullptr && blockIdx.x == 0;
    if (stamp && threadIdx.x == 0) {
        a.dbg[4000] = clock64();
    }
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < NT; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < NB; ++s) {
            mbar_init(bready_bar(s), NUM_DQ_WARPS);
            mbar_init(bfree_bar(s), 1);
        }
        mbar_init(accum_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    volatile int* abort_flag = &s_abort;

    if (warp == 0) {
        // ------------------------------------------------------------------ producer
        // (both issuing roles run converged with one elected lane: elect_one)
        const bool leader = elect_one();
        for (int it = 0; it < nkb; ++it) {
            const int s = it % NT, r = it / NT;
            if (!__all_sync(0xffffffffu, mbar_wait(empty_bar(s), (r & 1) ^ 1, abort_flag, a.status, (1 << 16) | it))) {
                break;
            }
            if (leader) {
                if (stamp && it < 1000) {
                    a.dbg[it] = clock64();
                }
                mbar_expect_tx(full_bar(s), mt_live * A_BYTES + nrbv * (TILE_WORDS * 4));
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    if (mt < mt_live) {
                        tma_load_2d(a_addr(s) + mt * A_BYTES, &tmap_x, (kb0 + it) * BK, m0 + mt * BM, full_bar(s));
                    }
                }
                // the tile's row blocks are contiguous at one k-block (k-block-major layout): one copy
                bulk_load(raw_addr(s), a.qt + ((size_t)(kb0 + it) * a.nrb_w + rb0) * TILE_WORDS,
                          nrbv * (TILE_WORDS * 4), full_bar(s));
            }
            __syncwarp();
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t idesc = (1u << 4) | ((uint32_t)(a.bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        const bool leader = elect_one();
        bool ok = true;
        for (int it = 0; it < nkb; ++it) {
            const int s = it % NT, r = it / NT, sb = it % NB, rb_ = it / NB;
            const bool in = mbar_wait(full_bar(s), r & 1, abort_flag, a.status, (2 << 16) | it) &&
                            mbar_wait(bready_bar(sb), rb_ & 1, abort_flag, a.status, (3 << 16) | it);
            ok = __all_sync(0xffffffffu, in);
            if (!ok) {
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t db = umma_desc(b_addr(sb));
            const uint64_t da0 = umma_desc(a_addr(s));
            if (leader) {
                if (stamp && it < 1000) {
                    a.dbg[3000 + it] = clock64();
                }
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    if (mt < mt_live) {
                        const uint64_t da = da0 + (uint64_t)(mt * A_BYTES >> 4);
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j) {
                            umma_f16(tmem + mt * 256, da + 2 * j, db + 2 * j, idesc, (it > 0 || j > 0) ? 1u : 0u);
                        }
                    }
                }
                umma_commit(empty_bar(s));
                umma_commit(bfree_bar(sb));
            }
            __syncwarp();
        }
        if (ok && leader) {
            umma_commit(accum_bar);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ dequantise, then epilogue
        const int dw = warp - 2;
        // bank-conflict-free assignment of the 32 (g,t) slots of a tile to lanes: g runs 0 3 4 7 | 1 2 5 6 over the quads, so
        // that the 16-byte reads of a quarter-warp and the 8-byte swizzled writes of a half-warp hit distinct banks
        const int t = lane & 3, g = (0x65217430u >> (4 * (lane >> 2))) & 7;
        const int ng = a.k / GROUP;
        bool ok = true;
        // scales of k-block `it` for this lane's two row blocks, fetched one k-block ahead
        auto load_scales = [&](int it, uint32_t (&sc)[2]) {
            sc[0] = sc[1] = 0;
            if (dw < nrbv && it < nkb) {
                const int kbi = kb0 + it;
                const uint32_t* sp = a.st + ((size_t)(rb0 + dw) * ng) * 8 + g;
                if (GROUP >= BK) {
                    sc[0] = sc[1] = __ldg(sp + (size_t)(kbi * BK / GROUP) * 8);
                } else {
                    sc[0] = __ldg(sp + (size_t)(kbi * 2) * 8);
                    sc[1] = __ldg(sp + (size_t)(kbi * 2 + 1) * 8);
                }
            }
        };
        uint32_t sc[2], sc_next[2];
        load_scales(0, sc_next);
        for (int it = 0; it < nkb && ok; ++it) {
            const int s = it % NT, r = it / NT, sb = it % NB, rb_ = it / NB;
            sc[0] = sc_next[0];
            sc[1] = sc_next[1];
            load_scales(it + 1, sc_next);
            ok = mbar_wait(full_bar(s), r & 1, abort_flag, a.status, (4 << 16) | it) &&
                 mbar_wait(bfree_bar(sb), (rb_ & 1) ^ 1, abort_flag, a.status, (6 << 16) | it);
            if (!ok) {
                break;
            }
            if (stamp && threadIdx.x == 64 && it < 1000) {
                a.dbg[1000 + it] = clock64();
            }
            {
                const int rbi = dw;
                if (rbi < nrbv) {
                    const uint4 raw = *reinterpret_cast<const uint4*>(
                        base_ptr + (raw_addr(s) - base) + rbi * (TILE_WORDS * 4) + (4 * g + t) * 16);
                    const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
                    const uint32_t row_off = b_addr(sb) + (uint32_t)(rbi * TILE_ROWS + g) * 128u;
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        uint32_t f[4];
                        dequant_word(rw[w], f);
                        const uint32_t s2 = sc[w >> 1];
                        const uint32_t s_r0 = __byte_perm(s2, s2, 0x1010);  // (s[r0], s[r0])
                        const uint32_t s_r1 = __byte_perm(s2, s2, 0x3232);  // (s[r1], s[r1])
                        const uint32_t piece = (uint32_t)(((2 * w + (t >> 1)) ^ g) << 4) + (uint32_t)(t & 1) * 8u;
                        *reinterpret_cast<uint2*>(base_ptr + (row_off - base) + piece) =
                            make_uint2(hmul2u(f[0], s_r0), hmul2u(f[2], s_r0));
                        *reinterpret_cast<uint2*>(base_ptr + (row_off - base) + 8u * 128u + piece) =
                            make_uint2(hmul2u(f[1], s_r1), hmul2u(f[3], s_r1));
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bready_bar(sb));
            }
            if (stamp && threadIdx.x == 64 && it < 1000) {
                a.dbg[2000 + it] = clock64();
            }
        }
        {
            // epilogue by all 16 warps: a warp may touch TMEM lanes 32*(warp%4) .. +31; the four warps of a
            // lane quadrant take every fourth 32-column chunk
            if (ok) {
                ok = mbar_wait(accum_bar, 0, abort_flag, a.status, (5 << 16));
            }
            ok = __all_sync(0xffffffffu, ok);
            if (stamp && threadIdx.x == 64) {
                a.dbg[4001] = clock64();
            }
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int quad = warp & 3;
                const int ncols = min(a.bn, a.n - n0);
                int n_staged = 0;
                for (int mc = 0; mc < mt_live * (BN / 32); ++mc) {
                    const int mt = mc / (BN / 32), c0 = (mc % (BN / 32)) * 32;
                    if (c0 >= ncols || (mc & 3) != (dw >> 2)) {
                        continue;
                    }
                    const int row_l = mt * BM + quad * 32 + lane;
                    const int row = m0 + row_l;
                    const float rw = (a.row_w != nullptr && row_l < rows_valid) ? a.row_w[row] : 1.0f;
                    // TMA-store path: every box of a dense tile (the tensor map clips at the batch's end); of a grouped
                    // tile only the boxes whose 32 rows all belong to the tile's expert segment
                    const bool staged_box = a.tma_store && ks == 1 && (!a.grouped || mt * BM + quad * 32 + 32 <= rows_valid);
                    uint32_t v[32];
                    tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(mt * 256 + c0), v);
                    if (ks > 1) {
                        // split-K: the f32 sums of this split go to scratch as they are
                        if (row_l < rows_valid) {
                            float4* pp = reinterpret_cast<float4*>(
                                a.part + ((size_t)sidx * ks + split) * (size_t)(BMT * BN) + (size_t)row_l * BN + c0);
#pragma unroll
                            for (int i = 0; i < 32; i += 4) {
                                if (c0 + i < ncols) {
                                    pp[i / 4] = make_float4(__uint_as_float(v[i]), __uint_as_float(v[i + 1]),
                                                            __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
                                }
                            }
                        }
                    } else if (a.glu && staged_box) {
                        // as below, through a staging tile of 32 rows x 16 outputs (32-byte rows, no swizzle)
                        uint32_t pk[8];
#pragma unroll
                        for (int i = 0; i < 16; i += 2) {
                            const __half h0 = silu_mul_f16(__uint_as_float(v[i]) * a.out_mul, __uint_as_float(v[16 + i]) * a.out_mul);
                            const __half h1 = silu_mul_f16(__uint_as_float(v[i + 1]) * a.out_mul, __uint_as_float(v[17 + i]) * a.out_mul);
                            pk[i / 2] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
                        }
                        if (n_staged >= 2) {
                            if (lane == 0) {
                                bulk_wait_group_read<1>();
                            }
                            __syncwarp();
                        }
                        const uint32_t sbuf = base + (uint32_t)dw * 8192u + (uint32_t)(n_staged & 1) * 4096u;
                        sts128(sbuf + (uint32_t)lane * 32u, make_uint4(pk[0], pk[1], pk[2], pk[3]));
                        sts128(sbuf + (uint32_t)lane * 32u + 16u, make_uint4(pk[4], pk[5], pk[6], pk[7]));
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tmap_y, sbuf, (n0 + c0) / 2, m0 + mt * BM + quad * 32);
                            bulk_commit_group();
                        }
                        ++n_staged;
                    } else if (a.glu) {
                        // a 32-column chunk = the gate sums and the up sums of the same 16 outputs
                        if (row_l < rows_valid && c0 < ncols) {
                            uint32_t pk[8];
#pragma unroll
                            for (int i = 0; i < 16; i += 2) {
                                const __half h0 = silu_mul_f16(__uint_as_float(v[i]) * a.out_mul, __uint_as_float(v[16 + i]) * a.out_mul);
                                const __half h1 = silu_mul_f16(__uint_as_float(v[i + 1]) * a.out_mul, __uint_as_float(v[17 + i]) * a.out_mul);
                                pk[i / 2] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
                            }
                            uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<__half*>(a.out) + (size_t)row * (a.n / 2) +
                                                                (n0 + c0) / 2);
                            o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                            o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                        }
                    } else if (staged_box) {
                        // The warp's 32 rows x 32 columns go to a staging tile in the (now idle) operand rings, laid out
                        // with the tensor map's swizzle so that the 16-byte writes of a quarter-warp hit distinct banks,
                        // and leave as one TMA store: whole 128-byte lines instead of 32 scattered half-sectors per
                        // instruction.  Rows past the batch and columns past n are clipped by the tensor map.  Two
                        // staging tiles per warp: the store of one is read out while the next is filled.
                        if (a.out_mul != 1.0f) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                v[i] = __float_as_uint(__uint_as_float(v[i]) * a.out_mul);
                            }
                        }
                        if (a.row_w != nullptr) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                v[i] = __float_as_uint(mul_row_w(__uint_as_float(v[i]), rw));
                            }
                        }
                        if (n_staged >= 2) {
                            if (lane == 0) {
                                bulk_wait_group_read<1>();
                            }
                            __syncwarp();
                        }
                        const uint32_t sbuf = base + (uint32_t)dw * 8192u + (uint32_t)(n_staged & 1) * 4096u;
                        if (a.out_f16) {
                            const uint32_t rowp = sbuf + (uint32_t)lane * 64u, sw = (uint32_t)(lane >> 1) & 3u;
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                uint4 pk;
                                __half2 h;
                                h = __floats2half2_rn(__uint_as_float(v[8 * c]), __uint_as_float(v[8 * c + 1]));
                                pk.x = *reinterpret_cast<uint32_t*>(&h);
                                h = __floats2half2_rn(__uint_as_float(v[8 * c + 2]), __uint_as_float(v[8 * c + 3]));
                                pk.y = *reinterpret_cast<uint32_t*>(&h);
                                h = __floats2half2_rn(__uint_as_float(v[8 * c + 4]), __uint_as_float(v[8 * c + 5]));
                                pk.z = *reinterpret_cast<uint32_t*>(&h);
                                h = __floats2half2_rn(__uint_as_float(v[8 * c + 6]), __uint_as_float(v[8 * c + 7]));
                                pk.w = *reinterpret_cast<uint32_t*>(&h);
                                sts128(rowp + (((uint32_t)c ^ sw) << 4), pk);
                            }
                        } else {
                            const uint32_t rowp = sbuf + (uint32_t)lane * 128u, sw = (uint32_t)lane & 7u;
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                sts128(rowp + (((uint32_t)c ^ sw) << 4), make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]));
                            }
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            if (m0 + mt * BM + quad * 32 < a.m) {   // a box wholly past the batch is not issued at all
                                tma_store_2d(&tmap_y, sbuf, n0 + c0, m0 + mt * BM + quad * 32);
                            }
                            bulk_commit_group();
                        }
                        ++n_staged;
                    } else if (row_l < rows_valid) {
                        if (a.out_mul != 1.0f) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                v[i] = __float_as_uint(__uint_as_float(v[i]) * a.out_mul);
                            }
                        }
                        if (a.row_w != nullptr) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                v[i] = __float_as_uint(mul_row_w(__uint_as_float(v[i]), rw));
                            }
                        }
                        if (a.out_f16) {
                            __half* o = reinterpret_cast<__half*>(a.out) + (size_t)row * a.n + n0 + c0;
#pragma unroll
                            for (int i = 0; i < 32; i += 8) {
                                if (c0 + i < ncols) {
                                    uint4 pk;
                                    __half2 h;
                                    h = __floats2half2_rn(__uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                                    pk.x = *reinterpret_cast<uint32_t*>(&h);
                                    h = __floats2half2_rn(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
                                    pk.y = *reinterpret_cast<uint32_t*>(&h);
                                    h = __floats2half2_rn(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5]));
                                    pk.z = *reinterpret_cast<uint32_t*>(&h);
                                    h = __floats2half2_rn(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7]));
                                    pk.w = *reinterpret_cast<uint32_t*>(&h);
                                    *reinterpret_cast<uint4*>(o + i) = pk;
                                }
                            }
                        } else {
                            float* o = reinterpret_cast<float*>(a.out) + (size_t)row * a.n + n0 + c0;
#pragma unroll
                            for (int i = 0; i < 32; i += 4) {
                                if (c0 + i < ncols) {
                                    *reinterpret_cast<uint4*>(o + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                                }
                            }
                        }
                    }
                }
                if (n_staged > 0) {
                    // the staging tiles must stay in place until the TMA stores have read them
                    if (lane == 0) {
                        bulk_wait_group_read<0>();
                    }
                    __syncwarp();
                }
            }
        }
    }

    if (stamp && threadIdx.x == 64) {
        a.dbg[4002] = clock64();
    }
    if (ks > 1) {
        __threadfence();   // this thread's partial sums, before the ticket below
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
    if (ks > 1) {
        // Every split of the tile adds a slice of its rows over all partial tiles, in split order (the same bits whatever
        // the arrival order), converts and stores.  One CTA adding all of them would read ksplit x 256 KB alone and take
        // longer than the wave it saves.  The splits of a tile are consecutive CTAs, at most 16 of them.  When every tile is
        // split there can be more CTAs than SMs; blocks start in the order of their index, so the earliest unfinished tile
        // has all of its splits on the GPU or next in line behind tiles that need nothing from it.  The wait for the
        // siblings is bounded all the same.  The ticket counts arrivals up to ksplit and departures up to 2 x ksplit, then
        // returns to zero.
        if (threadIdx.x == 0) {
            int ready = 0;
            if (!*abort_flag) {
                atomicAdd(a.counters + sidx, 1u);
                const long long t0 = clock64();
                ready = 1;
                while (*reinterpret_cast<volatile unsigned*>(a.counters + sidx) < (unsigned)ks) {
                    if (clock64() - t0 > (1ll << 31)) {
                        atomicCAS(a.status, 0, (7 << 16) | (sidx & 0xffff));   // a sibling split never arrived
                        ready = 0;
                        break;
                    }
                }
                __threadfence();
            }
            s_last = ready;
        }
        __syncthreads();
        if (s_last) {
            const int ncols = min(a.bn, a.n - n0), c4n = ncols / 4;
            const float* base_p = a.part + (size_t)sidx * ks * (size_t)(BMT * BN);
            const int r_begin = (int)((long long)rows_valid * split / ks), r_end = (int)((long long)rows_valid * (split + 1) / ks);
            for (int idx = threadIdx.x; idx < (r_end - r_begin) * c4n; idx += NUM_THREADS) {
                const int row_l = r_begin + idx / c4n, c = (idx % c4n) * 4;
                float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
                const float* src = base_p + (size_t)row_l * BN + c;
                for (int sp0 = 0; sp0 < ks; sp0 += 8) {
                    float4 pv[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {      // loads of up to eight splits in flight, then added in order
                        pv[q] = sp0 + q < ks ? __ldcg(reinterpret_cast<const float4*>(src + (size_t)(sp0 + q) * (BMT * BN)))
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        if (sp0 + q < ks) {
                            sum.x += pv[q].x;
                            sum.y += pv[q].y;
                            sum.z += pv[q].z;
                            sum.w += pv[q].w;
                        }
                    }
                }
                const int row = m0 + row_l;
                float o4[4] = {sum.x * a.out_mul, sum.y * a.out_mul, sum.z * a.out_mul, sum.w * a.out_mul};
                if (a.row_w != nullptr) {
                    const float rw = a.row_w[row];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        o4[i] = mul_row_w(o4[i], rw);
                    }
                }
                if (a.out_f16) {
                    const __half2 h0 = __floats2half2_rn(o4[0], o4[1]), h1 = __floats2half2_rn(o4[2], o4[3]);
                    uint2 pk;
                    pk.x = *reinterpret_cast<const uint32_t*>(&h0);
                    pk.y = *reinterpret_cast<const uint32_t*>(&h1);
                    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(a.out) + (size_t)row * a.n + n0 + c) = pk;
                } else {
                    *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + (size_t)row * a.n + n0 + c) =
                        make_float4(o4[0], o4[1], o4[2], o4[3]);
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                if (atomicAdd(a.counters + sidx, 1u) == 2u * (unsigned)ks - 1u) {
                    a.counters[sidx] = 0;   // every split has read what it needed: ready for the next launch
                }
            }
        }
    }
}

}  // namespace

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess) {
            fn = (EncodeTiledFn)p;
        }
    }
    return fn;
}

cudaError_t gemm_init_device() {
    cudaError_t e;
#define W4_SET(G, MTV) \
    e = cudaFuncSetAttribute(gemm_w4a16_tc_kernel<G, MTV>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<MTV>::SMEM); \
    if (e != cudaSuccess) return e;
    W4_SET(128, 1)
    W4_SET(128, 2)
    W4_SET(32, 1)
    W4_SET(32, 2)
#undef W4_SET
    return cudaSuccess;
}

// What the pairs without K splits were first estimated to take, when a stage of 128 channels took them 0.317 us and more (groups of 32: 0.445).  The
// estimate of gemm_ts2_choose has stages of half that.  This one still draws the line where that one is no guide: where pairs give up precision for
// time, and where calls had been theirs that the other, outside of what it was fitted to, would give away.
static double pairs_first_us(const Lin* l, int t, int out_kind, int sm_count) {
    const int n_tiles = (l->n + 255) / 256, stages = (l->k + 2 * BK - 1) / (2 * BK), pairs = sm_count / 2;
    double best = 1e30;
    for (int cap = 256; cap >= 96; cap -= 32) {
        const int m_tiles = (t + cap - 1) / cap, tok = ((t + m_tiles - 1) / m_tiles + 31) / 32 * 32;
        const long long tiles = (long long)m_tiles * n_tiles, waves = (tiles + pairs - 1) / pairs;
        const double full = std::min(1.0, std::max(0.0, ((double)tiles / (waves * pairs) - 0.41) / 0.52));
        const double light = std::max(l->group == 128 ? 0.317 : 0.445, 0.00224 * tok), heavy = std::max(l->group == 128 ? 0.439 : 0.470, 0.082 + 0.00254 * tok);
        const double f32 = out_kind == W4A16_OUT_F16 ? 0.0 : 0.0263 * tok - 3.23;
        best = std::min(best, 5.4 + waves * (stages * (light + std::max(0.0, heavy - light) * full) + f32) + (waves - 1) * 1.7);
    }
    return best;
}

int Dec::gemm(const Lin* l, const void* x, void* dst, int t, int out_kind, cudaStream_t st) {
    if (((uintptr_t)x & 15) != 0 || ((uintptr_t)dst & 15) != 0) {
        return fail("w4a16 gemm: x and dst must be 16-byte aligned");
    }
    if (tune_gemm_pair > 1) {
        const int ks = std::min(std::max(tune_gemm_pair_ks, 1), (l->k + 2 * TILE_K - 1) / (2 * TILE_K));
        return gemm_ts2(l, x, dst, t, out_kind, tune_gemm_pair, ks, ks > 1 || tune_gemm_pair_halves, st);
    }
    // Tile shape and K split are chosen together by a small cost model (microseconds, fitted to measurements on B200).  A
    // k-block takes 0.30 + 0.00105 bn with one 128-token block; with two, 0.295 + 0.00133 bn while at most 100 CTAs run and
    // 0.163 + 0.0024 bn (0.78 at 256) when the GPU is full; 5 us around a wave; a split tile another 3.5 us and, at 256 rows,
    // 0.065 us per token for writing, awaiting and adding f32 partial tiles.  Candidates per tile shape: whole tiles only;
    // whole tiles plus a split last wave; every tile split 2..16 ways (at least four k-blocks per split, partial tiles within
    // 128 MB of scratch).  Tiles narrower than 256 rows multiply less per expanded k-block and are taken where they fill SMs
    // that 256 leaves idle, by a tenth at least (1024 tokens, 5120 x 17408: 128 tiles of 160 rows 149 us, 80 of 256 178 us;
    // 5120 x 6144: 57 against 67 us).  224 rows never won the estimate over 20000 shapes and are there for the tuning key.
    const int nkb_all = l->k / BK;
    struct Choice {
        int mt, bn, n_whole, ks;
        double cost;
    };
    Choice best{1, BN, 0, 1, 1e30}, whole = best;     // of all candidates, of those without a split
    for (int bnc : {256, 224, 192, 160, 128}) {
        if (tune_gemm_bn > 0 ? bnc != tune_gemm_bn : (bnc != BN && tune_gemm_ksplit > 0)) {
            continue;
        }
        const int n_tiles = (l->n + bnc - 1) / bnc;
        const double bar = bnc == BN || tune_gemm_bn > 0 ? 1.0 : 1.0 / 0.9;     // what a narrow tile's estimate is weighed with
        for (int mtc = 1; mtc <= 2; ++mtc) {
            if ((tune_gemm_mt == 1 || tune_gemm_mt == 2) && mtc != tune_gemm_mt) {
                continue;
            }
            const int m_tiles = (t + BM * mtc - 1) / (BM * mtc);
            // a second, empty token block is neither fetched nor multiplied: its k-blocks cost what one block costs
            const bool two = mtc == 2 && t > BM;
            const long long tiles = (long long)m_tiles * n_tiles;
            const double tile_bytes = (double)BM * mtc * BN * 4.0;
            auto ctas_cost = [&](long long ctas, int nk, bool split) {
                const long long waves = ctas / sm_count, rest = ctas - waves * sm_count;
                const double around = 5.0 + (split ? 3.5 + 0.065 * std::min(t, BM * mtc) * bnc / BN : 0.0);
                const double full = two ? 0.163 + 0.0024 * bnc : 0.30 + 0.00105 * bnc;
                const double light = two ? 0.295 + 0.00133 * bnc : full;
                return waves * (nk * full + around) + (rest > 0 ? nk * (rest <= 100 ? light : full) + around : 0.0);
            };
            auto consider = [&](long long n_whole, int ks) {
                const long long split_tiles = tiles - n_whole;
                if (ks > 1 && (split_tiles > 4096 || split_tiles * ks * tile_bytes > 128.0 * (1 << 20))) {
                    return;
                }
                double c = ctas_cost(n_whole, nkb_all, false);
                if (split_tiles > 0) {
                    c += ctas_cost(split_tiles * ks, (nkb_all + ks - 1) / ks, ks > 1);
                }
                if (c * bar < best.cost) {
                    best = Choice{mtc, bnc, (int)n_whole, ks, c * bar};
                }
                if (ks == 1 && c * bar < whole.cost) {
                    whole = Choice{mtc, bnc, (int)n_whole, ks, c * bar};
                }
            };
            if (tune_gemm_ksplit > 0) {
                consider(0, std::min(tune_gemm_ksplit, std::max(1, nkb_all)));
                continue;
            }
            consider(tiles, 1);
            if (tune_gemm_ksplit < 0) {
                continue;
            }
            const long long rem = tiles % sm_count;
            if (rem > 0 && tiles > sm_count) {
                for (int ks = 2; ks <= 16 && nkb_all / ks >= 4; ++ks) {
                    consider(tiles - rem, ks);
                }
            }
            for (int ks = 2; ks <= 16 && nkb_all / ks >= 4; ++ks) {
                consider(0, ks);
            }
        }
    }
    // The weight-row form (gemm_ts.cu) takes the calls that it finishes sooner: up to about 128 tokens nearly all of them (its
    // MMA tile is as wide as the batch: 27 x 34816 x 5120 in 31 us against 52), above that those whose tiles here leave SMs
    // idle (512 x 7168 x 5120: 32 against 59 us); in full waves the 256 x 256 tiles are up to a fifth faster (256 x 34816 x
    // 5120: 67 against 72 us).  At a tie, within a tenth, this form; above 1024 tokens with K below 3072 within a fifth: there the
    // estimates leave out part of what the weight-row form's many short tiles cost.  Where its estimate is 0.8..0.9 of this
    // form's, at 1025..4096 tokens, it took 0.65..0.97 of the time on 24 shapes with K >= 3072 and 1.01 on two (1281 tokens, 7168
    // x 5120: 80 against 99 us, 5120 x 17408: 180 against 234), and 0.77..1.30 on 24 with a shorter K (1391 tokens, 15824 x 512:
    // 41 against 37 us; 2332 tokens, 22768 x 1216: 162 against 150); up to 1024 tokens 0.61..0.99 at any K (16 shapes).  More
    // than 4096 tokens were not compared: a fifth, too.
    const double bar_ts = t <= 1024 || (l->k >= 3072 && t <= 4096) ? 0.9 : 0.8;
    if (tune_gemm_form == 2 || (tune_gemm_form == 0 && tune_gemm_ksplit == 0 && tune_gemm_mt == 0 && tune_gemm_bn == 0)) {
        const TsChoice c = gemm_ts_choose(l->n, l->k, t);
        if (tune_gemm_form == 2 && c.tok == 0) {
            return fail("w4a16 gemm: no weight-row tile for %d x %d x %d (gemm_ts_ksplit=%d: no such cluster on this device)", t, l->n,
                        l->k, tune_ts_ks);
        }
        const bool ts = tune_gemm_form == 2 || c.cost < bar_ts * best.cost;
        const bool stays = ts && (c.ks > 1 ? l->k >= 16384 && t >= 256 : t <= 320 && (long long)l->n * l->k <= 1 << 20);
        if (t > 64 && t <= 4096 && !stays && tune_gemm_form == 0 && tune_gemm_pair == 0 && tune_ts_tok == 0 && tune_ts_ks == 0 &&
            tune_gemm_tma_store == 1) {
            // The pairs (gemm_ts2.cu) take f16 results that they are estimated to finish sooner.  The estimates of the weight-row form run 5 % high
            // in the median, so the line lies at 0.92 of them, 0.9 below 256 tokens, at 0.84 where they split K over clusters, and at 0.8 up to 128
            // tokens, where a wrong choice costs most.  Over 308 measured calls (22 shapes, 72..3000 tokens) the choice takes 1.0 % more than the
            // best form and tile of each; with a line that ended at split calls, and the estimates before it, it took 7.2 %.  Split calls of
            // K >= 16384 from 256 tokens on, and up to 320 tokens of linears of up to 2^20 weights, stay with the weight rows, as the tests name them
            // (256 x 5120 x 17408: 44 us, pairs of 96 tokens 40; 300 x 1024 x 1024: 5.0, 4.4).  Up to 64 and above 4096 tokens the pairs were not
            // compared.
            // The f32 results of such a call are what its f16 results are rounded from.  Where the weight rows would split K, results of either kind get the same
            // tiles, K splits and accumulators: the choice is made once, with the estimates for f16 results.  Otherwise f16 results come from pairs
            // without a K split, and f32 results from any form without one -- each of the three then adds the channels of a sum in the same order: the
            // form that they have without the pairs, unless that splits tiles: then the token-row form without a split, or the pairs where a nearly
            // empty last wave is what the split was for (its estimate leaves out that the full waves hold the clock down) or where they are ahead
            // by a clear margin (their estimate for f32 results is good to a tenth), or were by their first estimate.  f32, us with the split / without /
            // pairs: 7168 x 5120 at 4096 tokens 235 / 257 / 230, at 3000 185 / 218 / 170; 5120 x 17408 at 2048 269 / 314 / 256, at 4096 524 / 566 / 512;
            // 5120 x 6144 at 4096, 2.92 waves, 206 / 205 / 193.  Over 140 drawn calls the pairs took 0.36 to 0.93 of the tiles without a split; 12 of
            // them the margin alone would leave there (5632 x 8064 at 3517 tokens 253 / 225, 11120 x 9472 at 1183 194 / 174).
            const double line = t <= 128 ? 0.8 : !ts ? 0.98 : c.ks > 1 ? 0.84 : t < 256 ? 0.9 : 0.92;
            // In place of weight rows that split K: pairs whose accumulators take no more stages each (gemm_ts2), results of either kind from the
            // same tiles.  Below 256 tokens of more than 2^24 weights these may split K, too: few tiles (101 calls of both kinds take 0.89 of the time).
            // Smaller linears gain little or lose: 1792 x 5120 at 100 tokens 9.4 / 9.2 us, 4096 x 4096 11.1 / 10.8, 1024 x 4096 7.4 / 6.5; from 256
            // tokens on f32 results keep the forms that the tests name.
            // In place of token rows that split K, of every tile or of the last wave's: an accumulator drops what lies below its last bit, so the error grows
            // with the channels that go through one, and only the calls give up that split that did so from the first.  f32 error of the results' size
            // and us, token rows / pairs: 12400 x 20224 at 238 tokens 7.9e-6, 108 / 2.4e-5, 100; 720 x 15424 in groups of 32 at 2005 3.1e-6, 57.5 /
            // 1.8e-5, 41.8; 7168 x 17152 at 1521, a split last wave, 1.89e-5, 274 / 2.01e-5, 256.
            // In place of unsplit weight rows up to 16 stages long the estimates, which were fitted from 12 stages on, are no guide by themselves: their
            // launches take 2 us less than estimated, those of pairs no less.  us, weight rows / pairs: 11264 x 512 at 315 tokens 7.0 / 8.8, 3808 x 512 at
            // 250 4.3 / 5.2, 7344 x 896 at 82 5.2 / 5.9, 17664 x 1408 at 126 10.8 / 9.5.  Over 362 such calls the choice takes 1.1 % more than the better
            // form, without the 2 us 4.5 %.  Above 100 us the power limit holds the clock down, which the weight rows' estimate leaves out: 5296 x 6656 at
            // 2478 tokens 128 / 117, 10720 x 6400 at 1218 124 / 114; where the pairs are estimated at 0.92 to 0.95 of it they took 0.91 to 1.03 there, below
            // 100 us 0.98 to 1.06.
            auto unsplit_pairs = [&]() {
                const double p_us = gemm_ts2_choose(l, t, W4A16_OUT_F16, 1).cost, first = pairs_first_us(l, t, W4A16_OUT_F16, sm_count);
                if (!ts) {
                    return p_us < line * best.cost && (best.ks == 1 || first < 0.98 * best.cost);
                }
                return l->k <= 16 * 2 * BK ? p_us < c.cost - 2.0 || first < 0.98 * c.cost : p_us < (c.cost > 100.0 ? 0.98 : line) * c.cost;
            };
            if (ts && c.ks > 1) {
                const bool may_split = t < 256 && (long long)l->n * l->k > 16 << 20 && tune_gemm_pair_ks != 1;
                const TsChoice p = gemm_ts2_choose(l, t, W4A16_OUT_F16, may_split ? 4 : 1, c.ks);
                if (p.ks > 0 && p.cost < (p.ks > 1 ? 1.0 : line) * c.cost) {
                    return gemm_ts2(l, x, dst, t, out_kind, p.tok, p.ks, true, st);
                }
            } else if (unsplit_pairs()) {
                if (out_kind == W4A16_OUT_F16) {
                    return gemm_ts2(l, x, dst, t, out_kind, gemm_ts2_choose(l, t, out_kind, 1).tok, 1, false, st);
                }
                if (!ts && best.cost < whole.cost) {
                    const TsChoice p = gemm_ts2_choose(l, t, out_kind, 1);
                    const int rest = (t + BM * whole.mt - 1) / (BM * whole.mt) * ((l->n + whole.bn - 1) / whole.bn) % sm_count;
                    const bool empty = rest > 0 && rest <= 100;
                    if (p.cost < whole.cost * (empty ? 1.0 : 0.78) || pairs_first_us(l, t, out_kind, sm_count) < whole.cost * (empty ? 1.0 : 0.86)) {
                        return gemm_ts2(l, x, dst, t, out_kind, p.tok, 1, false, st);
                    }
                    best = whole;
                }
            }
        }
        if (ts) {
            return gemm_ts(l, x, dst, t, out_kind, c, st);
        }
    }
    const int bn = best.bn, n_tiles = (l->n + bn - 1) / bn;
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)l->k, (cuuint64_t)t};
    const cuuint64_t strides[1] = {(cuuint64_t)l->k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)BM};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr);
    }
    // the outputs as 32 x 32 boxes for the epilogue's TMA stores (f16: 64-byte rows, f32: 128-byte rows)
    CUtensorMap map_y = map;
    const bool out16 = out_kind == W4A16_OUT_F16;
    bool tma_store = tune_gemm_tma_store != 0;
    if (tma_store) {
        const cuuint64_t ydims[2] = {(cuuint64_t)l->n, (cuuint64_t)t};
        const cuuint64_t ystrides[1] = {(cuuint64_t)l->n * (out16 ? 2 : 4)};
        const cuuint32_t ybox[2] = {32, 32};
        cr = enc(&map_y, out16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, dst, ydims, ystrides,
                 ybox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, out16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                 CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) {
            tma_store = false;   // a refused map is not an error: the per-lane stores take any layout
        }
    }
    GemmArgs a;
    a.qt = l->qt;
    a.st = (const uint32_t*)l->st;
    a.out = dst;
    a.m = t;
    a.n = l->n;
    a.k = l->k;
    a.out_f16 = out16;
    a.n_tiles = n_tiles;
    a.bn = bn;
    const int mt = best.mt;
    a.m_tiles = (t + BM * mt - 1) / (BM * mt);
    a.nrb_w = l->n / TILE_ROWS;
    a.grouped = 0;
    a.tile_expert = a.tile_row0 = a.tile_rows = a.num_tiles = nullptr;
    a.expert0 = 0;
    a.row_w = nullptr;
    a.out_mul = l->out_mul;
    a.glu = 0;
    a.status = gemm_status;
    a.dbg = dbg_buf;
    a.tma_store = tma_store ? 1 : 0;
    const int tiles = a.m_tiles * a.n_tiles;
    int n_whole = best.n_whole, ks = best.ks;
    if (ks <= 1) {
        ks = 1;
        n_whole = tiles;
    }
    const size_t tile_floats = (size_t)BM * mt * BN;
    a.n_whole = n_whole;
    a.ksplit = ks;
    a.part = nullptr;
    a.counters = nullptr;
    if (ks > 1) {
        if (int rc = ensure_scratch((size_t)(tiles - n_whole) * ks * tile_floats, tiles - n_whole, st)) {
            return rc;
        }
        a.part = part;
        a.counters = counters;
    }
    const int grid = n_whole + (tiles - n_whole) * ks;
    if (l->group == 128) {
        if (mt == 2) {
            gemm_w4a16_tc_kernel<128, 2><<<grid, NUM_THREADS, Cfg<2>::SMEM, st>>>(map, map_y, a);
        } else {
            gemm_w4a16_tc_kernel<128, 1><<<grid, NUM_THREADS, Cfg<1>::SMEM, st>>>(map, map_y, a);
        }
    } else {
        if (mt == 2) {
            gemm_w4a16_tc_kernel<32, 2><<<grid, NUM_THREADS, Cfg<2>::SMEM, st>>>(map, map_y, a);
        } else {
            gemm_w4a16_tc_kernel<32, 1><<<grid, NUM_THREADS, Cfg<1>::SMEM, st>>>(map, map_y, a);
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        return cuda_fail("launch gemm", e);
    }
    last_kernel = "gemm_w4a16_tc_kernel<" + std::to_string(l->group) + "," + std::to_string(mt) + ">" +
                  (ks > 1 ? " split-K " + std::to_string(ks) + (n_whole > 0 ? " on the last wave" : "") : std::string());
    launches++;
    return 0;
}

// Grouped GEMM over expert segments: `l` stacks the local experts along n (n_per_expert rows each);
// xs holds the gathered rows (sorted by expert), the m-tile table lives on the device (moe.cu).
int Dec::gemm_grouped(const Lin* l, const void* xs, int xs_rows, void* out, int n_per_expert, const MoeBufs& b,
                      int max_tiles, const float* row_w, cudaStream_t st) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)l->k, (cuuint64_t)xs_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)l->k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)BM};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(xs), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr);
    }
    GemmArgs a;
    a.qt = l->qt;
    a.st = (const uint32_t*)l->st;
    a.out = out;
    a.m = xs_rows;
    a.n = n_per_expert;
    a.k = l->k;
    a.out_f16 = 1;
    a.m_tiles = max_tiles;
    a.n_tiles = (n_per_expert + BN - 1) / BN;
    a.bn = BN;
    a.nrb_w = l->n / TILE_ROWS;
    a.grouped = 1;
    a.tile_expert = b.tile_expert;
    a.tile_row0 = b.tile_row0;
    a.tile_rows = b.tile_rows;
    a.num_tiles = b.n_tiles;
    a.expert0 = moe.e0;
    a.row_w = row_w;
    a.out_mul = l->out_mul;
    a.glu = l->glu_f > 0 ? 1 : 0;
    a.n_whole = a.m_tiles * ((n_per_expert + BN - 1) / BN);
    a.ksplit = 1;
    a.part = nullptr;
    a.counters = nullptr;
    a.status = gemm_status;
    a.dbg = nullptr;
    // outputs as 32-row boxes for the TMA-store epilogue: [rows][n] f16, or [rows][n/2] f16 after the fused silu(gate)*up
    CUtensorMap map_y = map;
    a.tma_store = 0;
    if (tune_gemm_tma_store != 0) {
        const int n_out = a.glu ? n_per_expert / 2 : n_per_expert;
        const cuuint64_t ydims[2] = {(cuuint64_t)n_out, (cuuint64_t)xs_rows};
        const cuuint64_t ystrides[1] = {(cuuint64_t)n_out * 2};
        const cuuint32_t ybox[2] = {(cuuint32_t)(a.glu ? 16 : 32), 32};
        cr = enc(&map_y, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, out, ydims, ystrides, ybox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                 a.glu ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        a.tma_store = cr == CUDA_SUCCESS ? 1 : 0;   // else the per-lane stores
    }
    const int grid = a.m_tiles * a.n_tiles;
    if (l->group == 128) {
        gemm_w4a16_tc_kernel<128, 2><<<grid, NUM_THREADS, Cfg<2>::SMEM, st>>>(map, map_y, a);
    } else {
        gemm_w4a16_tc_kernel<32, 2><<<grid, NUM_THREADS, Cfg<2>::SMEM, st>>>(map, map_y, a);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        return cuda_fail("launch grouped gemm", e);
    }
    last_kernel = "gemm_w4a16_tc_kernel<" + std::to_string(l->group) + ",2> (grouped)";
    launches++;
    return 0;
}

}  // namespace w4
