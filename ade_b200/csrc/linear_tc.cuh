// One delta linear module  out = base + U^ (V^T x)  for up to 128 token rows, one launch, every contraction on the 5th-generation
// tensor cores.  The base term is either supplied (y_dense: what modules of 33-128 tokens take behind the library GEMM, in place of the
// reference's kernels A and B, src/kernels.py:486-886) or x W_b^T, streamed here (w_b: tall fused groups at 9-16 tokens).  Which calls come
// here is decided by ade_b200_linear_faster.
//
// The weights are the 128-row operand of tcgen05.mma (K-major, bf16), the token rows the N operand (padded to a multiple of 16), the
// accumulators stay in tensor memory for the whole launch.  Rows are cut into equal slices, one to three per SM, so that every SM streams
// and multiplies the same; every SM reads all of x (from L2).
//
// Everything a CTA multiplies goes through ONE ring of shared-memory stages (A part: up to 128 rows x 128 columns,
// B part: the token rows of the same columns), in this order:
//   A items   h = V^T x: the (rank group, 128-column block) pairs are dealt to all CTAs.  A = (code - zero) * scale, one bf16
//             rounding, written by the eight unpack warps; B = x by TMA.  The float32 partial sums of h go to scratch; when
//             all have arrived every CTA adds its share of the T x r elements, rounds to bf16 once and publishes it.
//   W items   the CTA's slices of W_b: A and B by TMA.  While the tensor core works through them, the unpack warps do the h
//             exchange above: the hand-overs are hidden under the stream as far as it is long enough.
//             (With a base term from the caller there are no W items; its values are added at the end.)
//   U items   U^ h on top of the same accumulators, 64 ranks at a time, spread over the end of the stream.  The scale of a (row, group) belongs to
//             the row, so it is multiplied into the A operand; scale (8 significant bits) times code - zero (4) is 12 bits,
//             which is exactly the sum of two bf16 values hi + lo: two MMA passes share one B tile of h and the product is
//             exact, as when the scale was applied to the float32 sums.
//
// What bounds it: with y_dense the chain of the two grid-wide hand-overs of h (partial sums visible, sums published: 3-5 us each under a
// loaded memory system) and of the U items behind them; with w_b the stream of W_b beside that chain.
// Measured (us per launch in a graph over rotated weights, warp-MMA kernel / this one).  Behind a given base term: 5000 x 5120 r = 896 T = 40
// 32.8 / 25.2, 4096 x 11008 r = 512 T = 100 42.4 / 26.6, 11008 x 4096 T = 128 52.9 / 25.7, 13824 x 5120 r = 640 T = 64 36.4 / 26.3, but 4096 x 4096
// r = 256 T = 64 16.0 / 16.1.  Base inside: 22016 x 4096 r = 1024 T = 16 60.5 / 45.8, r = 512 T = 12 44.4 / 40.0, 27648 x 5120 r = 1024 T = 16 86.2 / 59.5.
// One 64-column block per ring item took half as long again on tall slices (22016 x 4096 70): the issuing warp bound them.
#pragma once
#include <cuda.h>

#include "factored.cuh"
#include "recon.cuh"

namespace ade {

constexpr int LT_UNPACK_WARPS = 8;
constexpr int LT_LOAD_WARP = LT_UNPACK_WARPS;
constexpr int LT_MMA_WARP = LT_UNPACK_WARPS + 1;
constexpr int LT_THREADS = 32 * (LT_UNPACK_WARPS + 2);
constexpr int LT_UNPACK_THREADS = 32 * LT_UNPACK_WARPS;
constexpr int LT_TILE = 128;                       // rows of the MMA: ranks of a group, or up to 128 rows of a slice
constexpr int LT_KB = 64;                          // column block: 64 bf16 = one 128-byte swizzled row
constexpr int LT_ITEM = 2 * LT_KB;                 // columns of a ring item: one wait, one commit per two blocks (the issuing warp needs some
                                                   // 400 cycles per item, as long as the eight MMAs of a short slice take)
constexpr int LT_A_BLOCK = LT_TILE * 128;
constexpr int LT_A_BYTES = 2 * LT_A_BLOCK;
constexpr int LT_MAX_STAGES = 12;
constexpr int LT_MAX_SEG = 3;                      // slices per CTA (accumulators in tensor memory beside that of h)
constexpr int LT_MAX_BLOCKS = LT_MAX_SEG * 2 * 16;  // 64-rank blocks of a CTA at the highest rank
constexpr int LT_SMEM_FIXED = 1024 /* alignment */ + 8 * (2 * LT_MAX_STAGES + LT_MAX_BLOCKS + 3) + 32;

struct LinearParams {
    const uint8_t* uq;             // [M][r/2]
    const uint8_t* vt;             // [r][N/2]
    const uint16_t* us;            // [M][ng]
    const uint8_t* uz;             // [M][ng]
    const uint16_t* vs;            // [ng][N]
    const uint8_t* vz;             // [ng][N]
    __nv_bfloat16* h;              // scratch: bf16 [T][r]
    unsigned int* sync;            // scratch: [0] partial sums of h written, [1] CTAs past their waits, [3] shares of h published
    unsigned int* status;          // an expired wait records 1
    float* part;                   // workspace: [CTA][T][128] partial sums of h
    const __nv_bfloat16* y_dense;  // [T][M]: base term supplied by the caller, nothing of W_b is streamed; or nullptr
    __nv_bfloat16* out;            // [T][M]
    int T, tpad, M, N, r;
    int slices, segs;              // row slices, and how many of them a CTA takes
    int rows;                      // tallest slice
    int hparts;                    // CTAs per rank group in the computation of h
    int stages;
    int u_start;                   // W items a CTA streams before its first U item (h is there by then)
    uint32_t ring_bytes;
    uint32_t idesc;
    uint32_t tmem_cols;
    int n_blocks;                  // block-diagonal U^ as in FactoredParams
    int block_rows[5];
    int block_groups[5];
    long long spin_limit;
    int drop_arrivals;
};

struct LinearMaps {
    CUtensorMap w;                 // (M, N) bf16, box `rows` rows x 64, 128-byte swizzle
    CUtensorMap x;                 // (T, N) bf16, box tpad rows x 64, 128-byte swizzle
};

// D[tmem] (+)= A[smem desc] * B[smem desc], bf16 operands, float32 accumulate, K = 16
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t n) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ uint32_t bf2_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ void unpack_sync() { asm volatile("bar.sync 1, %0;" ::"n"(LT_UNPACK_THREADS) : "memory"); }

// Grid-wide wait of one thread for a counter (bounded; an expired wait is recorded and the launch carries on to its end).
__device__ __forceinline__ void lt_wait_count(const unsigned int* c, unsigned int want, const LinearParams& p, volatile int* abort_flag) {
    const long long t0 = clock64();
    while (ld_acquire_gpu(c) < want) {
        if (*abort_flag) return;
        if (clock64() - t0 > p.spin_limit) {
            *abort_flag = 1;
            atomicExch(p.status, 1u);
            return;
        }
    }
}

__global__ void __launch_bounds__(LT_THREADS, 1) linear_tc_kernel(const LinearParams p, const __grid_constant__ LinearMaps maps) {
    extern __shared__ uint8_t lt_smem[];
    const uint32_t raw0 = smem_u32(lt_smem);
    const uint32_t ring = (raw0 + 1023u) & ~1023u;
    const int S = p.stages;
    const uint32_t x_bytes = static_cast<uint32_t>(p.tpad) * 128u;               // one B block
    const uint32_t stage_bytes = LT_A_BYTES + 2 * x_bytes;
    const uint32_t bars = ring + p.ring_bytes;
    const uint32_t bar_full = bars, bar_empty = bars + 8 * S, bar_slot = bars + 16 * S, bar_h = bar_slot + 8 * LT_MAX_BLOCKS, bar_done = bar_h + 8,
                   bar_pass = bar_h + 16;
    uint8_t* gen = lt_smem + (bar_pass + 8 - raw0);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int G = gridDim.x, c = blockIdx.x;
    const int T = p.T, N = p.N, M = p.M, r = p.r, ng = r >> 7;
    const int kbs = N / LT_ITEM;                                 // items along the columns
    // A items: CTA c computes part c % hparts of rank group c / hparts
    const int hg = c / p.hparts, hp = c - hg * p.hparts;
    const bool has_h = hg < ng;
    const int a0 = has_h ? hp * kbs / p.hparts : 0;
    const int a1 = has_h ? (hp + 1) * kbs / p.hparts : 0;

    // The operands of the first A item are requested before anything else: their round trip runs under the set-up.
    struct AOp {
        uint4 q[2], s[8], z[4];
    } acur;
    const int row = tid >> 1, half = tid & 1;                    // operand row and half of the item an unpack thread writes
    auto fetch_a = [&](AOp& o, int kb) {
        const uint8_t* qrow = p.vt + static_cast<size_t>(hg * 128 + row) * (N >> 1) + half * 32 + kb * 64;
        const uint16_t* srow = p.vs + static_cast<size_t>(hg) * N + half * LT_KB + kb * LT_ITEM;
        const uint8_t* zrow = p.vz + static_cast<size_t>(hg) * N + half * LT_KB + kb * LT_ITEM;
#pragma unroll
        for (int j = 0; j < 2; ++j) o.q[j] = ldg16_stream(qrow + 16 * j);
#pragma unroll
        for (int j = 0; j < 8; ++j) o.s[j] = ldg16(srow + 8 * j);
#pragma unroll
        for (int j = 0; j < 4; ++j) o.z[j] = ldg16(zrow + 16 * j);
    };
    if (warp < LT_UNPACK_WARPS) {
        if (a0 < a1) fetch_a(acur, a0);
    }

    if (tid == LT_LOAD_WARP * 32) {
        for (int i = 0; i < S; ++i) {
            mbar_init(bar_full + 8 * i, 1 + LT_UNPACK_WARPS);
            mbar_init(bar_empty + 8 * i, 1);
        }
        for (int i = 0; i < LT_MAX_BLOCKS; ++i) mbar_init(bar_slot + 8 * i, 1);
        mbar_init(bar_h, 1);
        mbar_init(bar_done, 1);
        mbar_init(bar_pass, 1);
        *abort_flag = 0;
        fence_mbar_init();
        prefetch_tensormap(&maps.w);
        prefetch_tensormap(&maps.x);
    }
    if (warp == LT_MMA_WARP) {
        tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const WaitCtx wctx{abort_flag, reinterpret_cast<int*>(p.status), p.spin_limit};

    // W items: slices [slice0, slice0 + nseg)
    const int slice0 = c * p.segs;
    const int nseg = max(0, min(p.segs, p.slices - slice0));
    auto slice_row = [&](int s) { return static_cast<int>(static_cast<long long>(s) * M / p.slices); };
    // U items of segment s: the 64-rank blocks the slice's rows can touch
    auto u_range = [&](int s, int& u0, int& u1) {
        int lo = 0, hi = ng;
        if (p.n_blocks > 0) {
            const int m0 = slice_row(slice0 + s), m1 = slice_row(slice0 + s + 1);
            int l = ng, h = 0;
            for (int i = 0; i < p.n_blocks; ++i)
                if (p.block_rows[i] < m1 && p.block_rows[i + 1] > m0) {
                    l = min(l, p.block_groups[i]);
                    h = max(h, p.block_groups[i + 1]);
                }
            if (h > l) {
                lo = l;
                hi = h;
            }
        }
        u0 = 2 * lo;
        u1 = 2 * hi;
    };
    // The U items (one per 64-rank block) are spread evenly over the part of the W items that comes after u_start, so that their
    // preparation runs under the stream; a block of segment s comes after the segment's first W item, which starts the
    // accumulator.  Every role walks the same order: `u_before(j)` W items come before U block j.
    const int wtotal = p.y_dense ? 0 : nseg * kbs;
    int ucum[LT_MAX_SEG + 1] = {0, 0, 0, 0}, ufirst[LT_MAX_SEG] = {0, 0, 0};
#pragma unroll
    for (int s = 0; s < LT_MAX_SEG; ++s) {
        int u0 = 0, u1 = 0;
        if (s < nseg) u_range(s, u0, u1);
        ufirst[s] = u0;
        ucum[s + 1] = ucum[s] + u1 - u0;
    }
    const int ucount = ucum[LT_MAX_SEG];
    const int u_start = min(p.u_start, wtotal);
    auto u_seg = [&](int j) { return (j >= ucum[1]) + (j >= ucum[2]); };
    auto u_block = [&](int j) { return j < ucum[1] ? ufirst[0] + j : (j < ucum[2] ? ufirst[1] + j - ucum[1] : ufirst[2] + j - ucum[2]); };
    auto u_before = [&](int j) { return min(max(u_start + (j + 1) * (wtotal - u_start) / ucount, u_seg(j) * kbs + 1), wtotal); };

    if (warp == LT_LOAD_WARP) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 1;                                     // parity of the "empty" wait: the first round passes at once
            auto next = [&]() {
                if (++st == S) {
                    st = 0;
                    ph ^= 1;
                }
            };
            auto load_x = [&](int kb, uint32_t full) {
                tma_load_2d(ring + st * stage_bytes + LT_A_BYTES, &maps.x, kb * LT_ITEM, 0, full);
                tma_load_2d(ring + st * stage_bytes + LT_A_BYTES + x_bytes, &maps.x, kb * LT_ITEM + LT_KB, 0, full);
            };
            for (int kb = a0; kb < a1; ++kb, next()) {
                wait_bounded(bar_empty + 8 * st, ph, wctx, 1);
                mbar_arrive_expect_tx(bar_full + 8 * st, 2 * x_bytes);
                load_x(kb, bar_full + 8 * st);
            }
            const uint32_t w_bytes = static_cast<uint32_t>(p.rows) * 128u;
            int s = 0, kb = 0, m0 = slice_row(slice0), i = 0;
            for (int j = 0; j <= ucount; ++j) {
                const int stop = j < ucount ? u_before(j) : wtotal;
                for (; i < stop; ++i, next()) {
                    const uint32_t sa = ring + st * stage_bytes, full = bar_full + 8 * st;
                    wait_bounded(bar_empty + 8 * st, ph, wctx, 1);
                    mbar_arrive_n(full, LT_UNPACK_WARPS);        // the unpack warps have no part in a W item
                    mbar_arrive_expect_tx(full, 2 * (w_bytes + x_bytes));
                    tma_load_2d(sa, &maps.w, kb * LT_ITEM, m0, full);
                    tma_load_2d(sa + LT_A_BLOCK, &maps.w, kb * LT_ITEM + LT_KB, m0, full);
                    load_x(kb, full);
                    if (++kb == kbs) {
                        kb = 0;
                        m0 = slice_row(slice0 + ++s);
                    }
                }
                if (j < ucount) {                                // everything of a U item is written by the unpack warps, once its stage is free
                    wait_bounded(bar_empty + 8 * st, ph, wctx, 1);
                    mbar_arrive(bar_full + 8 * st);
                    mbar_arrive(bar_slot + 8 * j);
                    next();
                }
            }
            // Every CTA checks out once it is past its grid-wide waits; the last one re-arms the counters for the next call.  This
            // thread does it because nothing waits for it any more.
            wait_bounded(bar_pass, 0, wctx, 1);
            if (atomicAdd(p.sync + 1, 1u) == static_cast<unsigned int>(G - 1)) {
                atomicExch(p.sync, 0u);
                atomicExch(p.sync + 1, 0u);
                atomicExch(p.sync + 3, 0u);
            }
        }
        __syncwarp();
    } else if (warp == LT_MMA_WARP) {
        // ------------------------------------------------------------------ MMA issuer (warp-uniform loop, one elected lane)
        int st = 0;
        uint32_t ph = 0;
        auto next = [&]() {
            if (++st == S) {
                st = 0;
                ph ^= 1;
            }
        };
        auto mma4 = [&](uint32_t d, uint32_t a, uint32_t b, bool fresh) {
            const uint64_t ad = smem_desc_k_sw128(a), bd = smem_desc_k_sw128(b);
#pragma unroll
            for (int k = 0; k < 4; ++k) tc_mma_bf16(d, ad + 2 * k, bd + 2 * k, p.idesc, fresh && k == 0 ? 0u : 1u);
        };
        // a stage: both blocks of the columns, or (U item) the hi and lo parts of one 64-rank block against the same tile of h
        auto item = [&](uint32_t d, uint32_t b2, bool fresh) {
            const uint32_t sa = ring + st * stage_bytes, sb = sa + LT_A_BYTES;
            mma4(d, sa, sb, fresh);
            mma4(d, sa + LT_A_BLOCK, sb + b2, false);
            tc_commit(bar_empty + 8 * st);
        };
        for (int kb = a0; kb < a1; ++kb, next()) {
            wait_bounded(bar_full + 8 * st, ph, wctx, 1);
            tc_fence_after();
            if (elect_one()) {
                item(tmem_base, x_bytes, kb == a0);
                if (kb == a1 - 1) tc_commit(bar_h);
            }
            __syncwarp();
        }
        {
            uint32_t d = tmem_base + p.tpad;
            int kb = 0, i = 0;
            for (int j = 0; j <= ucount; ++j) {
                const int stop = j < ucount ? u_before(j) : wtotal;
                for (; i < stop; ++i, next()) {
                    wait_bounded(bar_full + 8 * st, ph, wctx, 1);
                    tc_fence_after();
                    if (elect_one()) item(d, x_bytes, kb == 0);
                    __syncwarp();
                    if (++kb == kbs) {
                        kb = 0;
                        d += p.tpad;
                    }
                }
                if (j < ucount) {
                    wait_bounded(bar_full + 8 * st, ph, wctx, 1);
                    tc_fence_after();
                    const int us = u_seg(j);
                    if (elect_one()) item(tmem_base + static_cast<uint32_t>(p.tpad) * (1 + us), 0u, wtotal == 0 && j == ucum[us]);
                    __syncwarp();
                    next();
                }
            }
        }
        if (elect_one()) tc_commit(bar_done);
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ unpack, h exchange, epilogue
        {
            int st = 0;
            uint32_t ph = 1;
            for (int kb = a0; kb < a1; ++kb) {
                wait_bounded(bar_empty + 8 * st, ph, wctx, 1);
                const uint32_t cw[8] = {acur.q[0].x, acur.q[0].y, acur.q[0].z, acur.q[0].w, acur.q[1].x, acur.q[1].y, acur.q[1].z, acur.q[1].w};
                const uint32_t dst = ring + st * stage_bytes + half * LT_A_BLOCK + static_cast<uint32_t>(row) * 128u;
#pragma unroll
                for (int wi = 0; wi < 8; ++wi) {                 // (code - zero) is exact; one rounding in the product
                    uint32_t e[4];
                    unpack8_bf16(cw[wi], e);
                    const uint4 zq = acur.z[wi >> 1];
                    const uint32_t z0 = (wi & 1) ? zq.z : zq.x, z1 = (wi & 1) ? zq.w : zq.y;
                    uint32_t o[4];
                    o[0] = bf2_mul(bf2_sub(e[0], __byte_perm(z0, 0x43434343u, 0x4140)), acur.s[wi].x);
                    o[1] = bf2_mul(bf2_sub(e[1], __byte_perm(z0, 0x43434343u, 0x4342)), acur.s[wi].y);
                    o[2] = bf2_mul(bf2_sub(e[2], __byte_perm(z1, 0x43434343u, 0x4140)), acur.s[wi].z);
                    o[3] = bf2_mul(bf2_sub(e[3], __byte_perm(z1, 0x43434343u, 0x4342)), acur.s[wi].w);
                    sts16(dst + ((wi ^ (row & 7)) << 4), make_uint4(o[0], o[1], o[2], o[3]));
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * st);
                if (kb + 1 < a1) fetch_a(acur, kb + 1);
                if (++st == S) {
                    st = 0;
                    ph ^= 1;
                }
            }
        }

        // ---- partial sums of h: tensor memory -> scratch, [part][token][rank]
        const int q = warp & 3, hcol = warp >> 2;                // tensor-memory lane quarter, column half
        const int rr = q * 32 + lane;                            // accumulator row of this thread
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        float* const part = p.part + static_cast<size_t>(c) * T * 128 + rr;
        if (a0 < a1) {
            wait_bounded(bar_h, 0, wctx, 1);
            tc_fence_after();
            for (int c0 = hcol * 16; c0 < p.tpad; c0 += 32) {
                uint32_t v[16];
                tmem_ld16_sync(lane_addr + c0, v);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (c0 + i < T) __stcg(part + static_cast<size_t>(c0 + i) * 128, __uint_as_float(v[i]));
            }
        }

        // Operands of the U blocks, one block ahead of their use: 32 codes of one row per thread, and 16-byte pieces of h.
        struct UOp {
            uint4 q;
            uint32_t s, z;
        } u, un;
        auto fetch_u = [&](UOp& o, int j) {
            const int s = slice0 + u_seg(j), kb = u_block(j);
            const int m = min(slice_row(s) + row, slice_row(s + 1) - 1);              // rows past the slice: any values, never stored
            o.q = ldg16_stream(p.uq + static_cast<size_t>(m) * (r >> 1) + half * 16 + kb * 32);
            o.s = p.us[static_cast<size_t>(m) * ng + (kb >> 1)];
            o.z = p.uz[static_cast<size_t>(m) * ng + (kb >> 1)];
        };
        auto fetch_h = [&](uint4 (&o)[4], int j) {
            const __nv_bfloat16* src = p.h + u_block(j) * 64 + (tid & 7) * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if ((tid >> 3) + 32 * i < T) o[i] = ldcg16(src + static_cast<size_t>((tid >> 3) + 32 * i) * r);
        };

        unpack_sync();
        if (tid == 0 && a0 < a1 && !p.drop_arrivals) red_release_gpu_add(p.sync, 1u);
        const bool by_warp = p.y_dense && T <= 64;
        if (!by_warp && ucount > 0) fetch_u(u, 0);                           // after the release: the fence in it would wait for these loads too
        if (tid == 0) lt_wait_count(p.sync, static_cast<unsigned int>(ng * p.hparts), p, abort_flag);
        unpack_sync();
        // ---- this CTA's share of h: four lanes per four ranks, each adds every fourth part, fixed order
        {
            const int quads = (T * r) >> 2;
            const int q0 = static_cast<int>(static_cast<long long>(c) * quads / G), q1 = static_cast<int>(static_cast<long long>(c + 1) * quads / G);
            const int sub = tid & 3;
            const size_t stride = static_cast<size_t>(T) * 128;
            for (int base = q0; base < q1; base += LT_UNPACK_THREADS / 4) {
                const int i = base + (tid >> 2);
                const bool live = i < q1;
                const int e = 4 * i, t = e / r, k = e - t * r;
                const float* src = p.part + (static_cast<size_t>(k >> 7) * p.hparts * T + t) * 128 + (k & 127);
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
                for (int j = sub; live && j < p.hparts; j += 40) {
                    uint4 a[10];
#pragma unroll
                    for (int k2 = 0; k2 < 10; ++k2) a[k2] = j + 4 * k2 < p.hparts ? ldcg16(src + (j + 4 * k2) * stride) : make_uint4(0, 0, 0, 0);
#pragma unroll
                    for (int k2 = 0; k2 < 10; ++k2) {
                        s0 += __uint_as_float(a[k2].x);
                        s1 += __uint_as_float(a[k2].y);
                        s2 += __uint_as_float(a[k2].z);
                        s3 += __uint_as_float(a[k2].w);
                    }
                }
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    s0 += __shfl_xor_sync(0xFFFFFFFFu, s0, o);
                    s1 += __shfl_xor_sync(0xFFFFFFFFu, s1, o);
                    s2 += __shfl_xor_sync(0xFFFFFFFFu, s2, o);
                    s3 += __shfl_xor_sync(0xFFFFFFFFu, s3, o);
                }
                if (live && sub == 0) {
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(s0, s1), hi = __floats2bfloat162_rn(s2, s3);
                    uint2 v;
                    v.x = *reinterpret_cast<const uint32_t*>(&lo);
                    v.y = *reinterpret_cast<const uint32_t*>(&hi);
                    *reinterpret_cast<uint2*>(p.h + e) = v;
                }
            }
        }
        unpack_sync();
        if (tid == 0) {
            red_release_gpu_add(p.sync + 3, 1u);
            lt_wait_count(p.sync + 3, static_cast<unsigned int>(G), p, abort_flag);
            mbar_arrive(bar_pass);                               // the load warp checks out for this CTA
        }
        unpack_sync();

        // ---- U items.  The load warp, which follows the ring item by item, says when a block's stage is free (one barrier per block: a
        // wait of this role's own on bar_empty could take an older phase of the same parity for the right one).
        if (by_warp) {
            // Nothing streams beside them, slices are short and h is small: a warp per block, so that the blocks' round trips for h
            // overlap (4096 x 4096 r = 512, this launch at T = 17 22.0 -> 17.7 us; from 65 tokens up one warp's share of h takes longer
            // than the round trips, T = 100 26.3 -> 29.4).
            for (int j = warp; j < ucount; j += LT_UNPACK_WARPS) {
                const int s = slice0 + u_seg(j), kb = u_block(j), m0 = slice_row(s), m1 = slice_row(s + 1);
                uint4 q8[8];
                uint32_t s8[8], z8[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (16 * k < p.rows) {
                        const int m = min(m0 + (lane >> 1) + 16 * k, m1 - 1);          // rows past the slice: any values, never stored
                        q8[k] = ldg16_stream(p.uq + static_cast<size_t>(m) * (r >> 1) + (lane & 1) * 16 + kb * 32);
                        s8[k] = p.us[static_cast<size_t>(m) * ng + (kb >> 1)];
                        z8[k] = p.uz[static_cast<size_t>(m) * ng + (kb >> 1)];
                    }
                const int us = ((a1 - a0) + j) % S;
                const uint32_t ua = ring + us * stage_bytes, hb = ua + LT_A_BYTES;
                wait_bounded(bar_slot + 8 * j, 0, wctx, 1);
                for (int tb = 0; tb < T; tb += 32) {
                    uint4 hv[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int t = tb + (lane >> 3) + 4 * k;
                        if (t < T) hv[k] = ldcg16(p.h + static_cast<size_t>(t) * r + kb * 64 + (lane & 7) * 8);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int t = tb + (lane >> 3) + 4 * k;
                        if (t < T) sts16(hb + t * 128 + (((lane & 7) ^ (t & 7)) << 4), hv[k]);
                    }
                }
#pragma unroll
                for (int k8 = 0; k8 < 8; ++k8) {
                    if (16 * k8 >= p.rows) break;
                    const int ur = (lane >> 1) + 16 * k8;
                    const uint32_t zz = kBf2_128 | z8[k8] | (z8[k8] << 16), s2 = s8[k8] | (s8[k8] << 16);
                    const uint32_t cw[4] = {q8[k8].x, q8[k8].y, q8[k8].z, q8[k8].w};
#pragma unroll
                    for (int wi = 0; wi < 4; ++wi) {
                        uint32_t e[4], hi[4], lo[4];
                        unpack8_bf16(cw[wi], e);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t dz = bf2_sub(e[k], zz);           // as below
                            hi[k] = bf2_mul(dz, s2);
                            lo[k] = bf2_fma(dz, s2, hi[k] ^ 0x80008000u);
                        }
                        const uint32_t off = ur * 128 + ((((lane & 1) * 4 + wi) ^ (ur & 7)) << 4);
                        sts16(ua + off, make_uint4(hi[0], hi[1], hi[2], hi[3]));
                        sts16(ua + LT_A_BLOCK + off, make_uint4(lo[0], lo[1], lo[2], lo[3]));
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive_n(bar_full + 8 * us, LT_UNPACK_WARPS);          // one warp for all eight
            }
        } else {
            // All eight warps on each block, operands one block ahead.
            uint4 hc[4], hn[4];
            if (ucount > 0) fetch_h(hc, 0);
            for (int j = 0; j < ucount; ++j) {
                if (j + 1 < ucount) {
                    fetch_u(un, j + 1);
                    fetch_h(hn, j + 1);
                }
                const int us = ((a1 - a0) + u_before(j) + j) % S;      // the block's stage
                wait_bounded(bar_slot + 8 * j, 0, wctx, 1);
                const uint32_t ua = ring + us * stage_bytes, hb = ua + LT_A_BYTES;
#pragma unroll
                for (int i = 0; i < 4; ++i) {                    // B tile: h of 64 ranks
                    const int t = (tid >> 3) + 32 * i, k8 = tid & 7;
                    if (t < T) sts16(hb + t * 128 + ((k8 ^ (t & 7)) << 4), hc[i]);
                }
                if (row < p.rows) {
                    const uint32_t zz = kBf2_128 | u.z | (u.z << 16), s2 = u.s | (u.s << 16);
                    const uint32_t cw[4] = {u.q.x, u.q.y, u.q.z, u.q.w};
#pragma unroll
                    for (int wi = 0; wi < 4; ++wi) {
                        uint32_t e[4], hi[4], lo[4];
                        unpack8_bf16(cw[wi], e);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t dz = bf2_sub(e[k], zz);           // exact
                            hi[k] = bf2_mul(dz, s2);                         // the product's upper 8 bits
                            lo[k] = bf2_fma(dz, s2, hi[k] ^ 0x80008000u);    // the rest of its 12, exact
                        }
                        const uint32_t off = row * 128 + (((half * 4 + wi) ^ (row & 7)) << 4);
                        sts16(ua + off, make_uint4(hi[0], hi[1], hi[2], hi[3]));
                        sts16(ua + LT_A_BLOCK + off, make_uint4(lo[0], lo[1], lo[2], lo[3]));
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * us);
                u = un;
#pragma unroll
                for (int i = 0; i < 4; ++i) hc[i] = hn[i];
            }
        }

        // ---- epilogue
        for (int s = 0; s < nseg; ++s) {
            const int m = slice_row(slice0 + s) + rr;
            const bool live = m < slice_row(slice0 + s + 1);
            uint32_t y[4][16];                               // base term, requested before the last products are waited for
            if (p.y_dense) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int t = hcol * 16 + 32 * k + i;
                        y[k][i] = live && t < T ? static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(p.y_dense) + static_cast<size_t>(t) * M + m)) : 0u;
                    }
            }
            if (s == 0) {
                wait_bounded(bar_done, 0, wctx, 1);
                tc_fence_after();
            }
            if (q * 32 >= p.rows) continue;                  // uniform in the warp
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c0 = hcol * 16 + 32 * k;
                if (c0 >= p.tpad) break;
                uint32_t v[16];
                tmem_ld16_sync(lane_addr + static_cast<uint32_t>(p.tpad) * (1 + s) + c0, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float o = __uint_as_float(v[i]);
                    if (p.y_dense) o += __uint_as_float(y[k][i] << 16);
                    if (live && c0 + i < T) p.out[static_cast<size_t>(c0 + i) * M + m] = __float2bfloat16_rn(o);
                }
            }
        }
    }

    drain_after_abort(abort_flag);
    tc_fence_before();
    __syncthreads();
    if (warp == LT_MMA_WARP) tmem_dealloc(tmem_base, p.tmem_cols);
}

// How a launch is cut: equal row slices, `segs` of them per CTA.
struct LinearSplit {
    int slices, segs, rows, stages, u_start;
    uint32_t ring_bytes;
};
constexpr int kLtRingMax = 232448 - LT_SMEM_FIXED;

inline bool linear_split(int M, int T, int tpad, int grid, LinearSplit& out) {
    LinearSplit s = {};
    s.segs = (M + LT_TILE * grid - 1) / (LT_TILE * grid);
    if (s.segs > LT_MAX_SEG) return false;
    s.slices = grid * s.segs;
    if (s.slices > M) s.slices = M;
    s.rows = (M + s.slices - 1) / s.slices;
    const int stage = LT_A_BYTES + 2 * tpad * 128;
    s.stages = kLtRingMax / stage;
    if (s.stages > LT_MAX_STAGES) s.stages = LT_MAX_STAGES;
    // h is there after about 10 us (two grid-wide hand-overs; more with more of it to add up); by then an SM has streamed this many items
    // (its share of 6.4 TB/s, or 0.34 us each).  U items that come up earlier would hold the stream up.
    const double item = s.rows * 256.0 * grid / 6.4e6 > 0.34 ? s.rows * 256.0 * grid / 6.4e6 : 0.34;
    s.u_start = static_cast<int>((10.0 + 0.04 * T) / item) + 1;
    s.ring_bytes = static_cast<uint32_t>(s.stages * stage);
    if (s.stages < 2) return false;
    out = s;
    return true;
}

// Workspace: partial sums of h.
inline size_t linear_workspace_bytes(int T, int grid) { return static_cast<size_t>(grid) * T * 128 * sizeof(float); }

}  // namespace ade
