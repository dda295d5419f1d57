// Producer side of the packed-delta format on the GPU: one pass from a factor of the truncated SVD to 4-bit codes,
// bfloat16 scales and zero-points.
//
// Replaces, for one factor X (rows x r, float32), the chain of src/quantization.py:244-285:
//     X * sqrt(S)                      (:266-268)
//     ... @ H                          (:270-272; H = normalised Sylvester Hadamard when r is a power of two, :56-70)
//     quantize_rowwise / _colwise      (:134-199, with _pin_zero_in_range :109-131)
// The reference multiplies by a dense r x r matrix (2 r^2 flops per row) and then makes about ten elementwise passes
// over the result.  Here a warp keeps a row in its registers (lane l holds elements 128 j + 4 l .. 4 l + 3 of every group j),
// applies the Hadamard rotation as a fast Walsh-Hadamard transform (r log2 r additions: the strides 1 and 2 and those of 128
// and above inside a thread, the five between with shuffles) and quantises its groups in place, so X is read once with
// 16-byte loads and codes, scales and zero-points are written once (5 bytes of traffic per element).  No barrier is needed
// for a row; without a rotation the groups are independent and every group is a "row" of 128.
//
// Both factors are "rows x r" here: U is (d_o, r); V is (d_i, r), and H^T (sqrt(S) V^T) = ((V sqrt(S)) H)^T for any
// H, so the V side runs the same row code with its outputs written transposed (codes (r, d_i), scales and
// zero-points (r/128, d_i)), 32 rows of a CTA at a time through shared memory so that the transposed writes are 32-byte
// segments.
//
// The quantisation arithmetic is the reference's, operation for operation in float32 (IEEE division, round half to
// even), so given the same rotated input the outputs are bit-identical to quantize_rowwise / quantize_colwise.  The
// transform sums in another order than a dense matmul, so after a rotation codes can differ by one step where a value
// sits on a rounding boundary.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ade {

constexpr int CQ_THREADS = 256;
constexpr int CQ_WARPS = CQ_THREADS / 32;
constexpr int CQ_ROWS = 32;            // rows per CTA (one transposed write segment)
constexpr int CQ_MAX_RANK = 2048;

// codes [CQ_ROWS][r + 4] (the padding spreads the transposing reads over the banks), then scales and zero-points [2 ng][CQ_ROWS]
__host__ __device__ inline size_t compress_smem_bytes(int r, bool transposed) {
    return transposed ? static_cast<size_t>(r + 4) * CQ_ROWS + static_cast<size_t>(r / 128) * CQ_ROWS * 4 : 0;
}

// Quantises one group of 128 held four values per lane.  Every operation rounds as the reference's float32 arithmetic does.
__device__ __forceinline__ uint32_t quantize_group(const float (&v)[4], float& sc, float& zp) {
    float lo = 3.402823466e38f, hi = -3.402823466e38f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        lo = fminf(lo, v[i]);
        hi = fmaxf(hi, v[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    if (lo == 0.f && hi == 0.f) {                                       // an all-zero group quantises as [-1, 1]
        lo = -1.f;
        hi = 1.f;
    }
    sc = __fdiv_rn(fmaxf(__fsub_rn(hi, lo), 1e-5f), 15.f);
    zp = rintf(__fdiv_rn(-lo, sc));
    if (zp < 0.f) {                                                     // one-signed groups are widened to contain 0
        sc = __fdiv_rn(fmaxf(hi, 1e-5f), 15.f);
        zp = 0.f;
    } else if (zp > 15.f) {
        sc = __fdiv_rn(fmaxf(-lo, 1e-5f), 15.f);
        zp = 15.f;
    }
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float q = fminf(fmaxf(__fadd_rn(rintf(__fdiv_rn(v[i], sc)), zp), 0.f), 15.f);
        c |= static_cast<uint32_t>(static_cast<uint8_t>(q)) << (8 * i);
    }
    return c;
}

// X (rows, r) float32; sqrt_s (r) float32 or nullptr.  ROT: a row of r = 128 NJ elements is rotated (Hadamard, r a power of two);
// otherwise NJ is 1 and the groups of a row are taken one by one.  VEC: X and sqrt_s are 16-byte aligned and codes 4-byte.
// Row-wise outputs: codes (rows, r), scale / zero (rows, r/128).  Transposed: codes (r, rows), scale / zero (r/128, rows).
// r = 512: 11008 rows 18.5 us, 4096 rows transposed 11.8 us (2.2 TB/s; about half of it issue-bound on shuffles and IEEE divisions).
// One row per CTA in shared memory with a barrier after every butterfly stride took about 170 us for the two.
template <int NJ, bool ROT, bool TRANSPOSED, bool VEC>
__global__ void __launch_bounds__(CQ_THREADS) compress_rows_kernel(const float* __restrict__ X, const float* __restrict__ sqrt_s,
                                                                     uint8_t* __restrict__ codes, __nv_bfloat16* __restrict__ scale,
                                                                     __nv_bfloat16* __restrict__ zero, int rows, int r) {
    extern __shared__ uint8_t cq_smem[];
    const int ng = r >> 7, pitch = r + 4;
    __nv_bfloat16* stile = reinterpret_cast<__nv_bfloat16*>(cq_smem + static_cast<size_t>(pitch) * CQ_ROWS);   // [2 ng][CQ_ROWS]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float norm = ROT ? rsqrtf(static_cast<float>(r)) : 1.0f;     // exact for r = 4^k, else within rsqrtf's 2 ulp of 1 / sqrt(r)
    const int m0 = blockIdx.x * CQ_ROWS;
    const int nrows = min(CQ_ROWS, rows - m0);
    const int parts = ROT ? 1 : ng;                                     // pieces a row is taken in
    for (int w = warp; w < nrows * parts; w += CQ_WARPS) {
        const int rr = ROT ? w : w / parts, g0 = ROT ? 0 : w - rr * parts;
        const size_t m = static_cast<size_t>(m0 + rr);
        const float* src = X + m * r + g0 * 128 + lane * 4;
        float v[NJ][4];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            if (VEC) {
                const float4 t = __ldcs(reinterpret_cast<const float4*>(src + 128 * j));
                v[j][0] = t.x;
                v[j][1] = t.y;
                v[j][2] = t.z;
                v[j][3] = t.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[j][i] = src[128 * j + i];
            }
        }
        if (sqrt_s) {
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const float* ss = sqrt_s + (g0 + j) * 128 + lane * 4;
                if (VEC) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(ss));
                    v[j][0] = __fmul_rn(v[j][0], t.x);
                    v[j][1] = __fmul_rn(v[j][1], t.y);
                    v[j][2] = __fmul_rn(v[j][2], t.z);
                    v[j][3] = __fmul_rn(v[j][3], t.w);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[j][i] = __fmul_rn(v[j][i], ss[i]);
                }
            }
        }
        if (ROT) {
            // butterflies of stride 1, 2 (registers), 4 .. 64 (lanes), 128 .. r / 2 (registers), in this order
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const float a = __fadd_rn(v[j][0], v[j][1]), b = __fsub_rn(v[j][0], v[j][1]);
                const float c = __fadd_rn(v[j][2], v[j][3]), d = __fsub_rn(v[j][2], v[j][3]);
                v[j][0] = __fadd_rn(a, c);
                v[j][1] = __fadd_rn(b, d);
                v[j][2] = __fsub_rn(a, c);
                v[j][3] = __fsub_rn(b, d);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float sign = (lane & o) ? -1.f : 1.f;             // other + mine, or other - mine: one rounding either way
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[j][i] = __fmaf_rn(v[j][i], sign, __shfl_xor_sync(0xFFFFFFFFu, v[j][i], o));
            }
#pragma unroll
            for (int h = 1; h < NJ; h <<= 1)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    if (!(j & h)) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float a = v[j][i], b = v[j + h][i];
                            v[j][i] = __fadd_rn(a, b);
                            v[j + h][i] = __fsub_rn(a, b);
                        }
                    }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int g = g0 + j, k = g * 128 + lane * 4;
            if (ROT) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[j][i] = __fmul_rn(v[j][i], norm);
            }
            float sc, zp;
            const uint32_t c = quantize_group(v[j], sc, zp);
            if (TRANSPOSED) {
                *reinterpret_cast<uint32_t*>(cq_smem + rr * pitch + k) = c;
                if (lane == 0) {
                    stile[g * CQ_ROWS + rr] = __float2bfloat16_rn(sc);
                    stile[(ng + g) * CQ_ROWS + rr] = __float2bfloat16_rn(zp);
                }
            } else {
                if (VEC) {
                    *reinterpret_cast<uint32_t*>(codes + m * r + k) = c;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) codes[m * r + k + i] = static_cast<uint8_t>(c >> (8 * i));
                }
                if (lane == 0) {
                    scale[m * ng + g] = __float2bfloat16_rn(sc);
                    zero[m * ng + g] = __float2bfloat16_rn(zp);
                }
            }
        }
    }
    if (TRANSPOSED) {
        __syncthreads();
        // A thread turns a 4 x 4 block of codes: four rows of the tile in, one word for each of four output rows.  Eight lanes
        // cover the 32 columns of an output row.
        const int rq = (threadIdx.x & 7) * 4;
        for (int kq = threadIdx.x >> 3; kq < (r >> 2); kq += CQ_THREADS / 8) {
            uint32_t a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const uint32_t*>(cq_smem + (rq + i) * pitch + 4 * kq);
            const uint32_t lo01 = __byte_perm(a[0], a[1], 0x5140), hi01 = __byte_perm(a[0], a[1], 0x7362);
            const uint32_t lo23 = __byte_perm(a[2], a[3], 0x5140), hi23 = __byte_perm(a[2], a[3], 0x7362);
            const uint32_t o[4] = {__byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632), __byte_perm(hi01, hi23, 0x5410),
                                   __byte_perm(hi01, hi23, 0x7632)};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint8_t* dst = codes + static_cast<size_t>(4 * kq + i) * rows + m0 + rq;
                if (nrows == CQ_ROWS && (rows & 3) == 0) {
                    *reinterpret_cast<uint32_t*>(dst) = o[i];
                } else {
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        if (rq + b < nrows) dst[b] = static_cast<uint8_t>(o[i] >> (8 * b));
                }
            }
        }
        for (int e = threadIdx.x; e < ng * CQ_ROWS; e += CQ_THREADS) {
            const int g = e / CQ_ROWS, rr = e % CQ_ROWS;
            if (rr < nrows) {
                scale[static_cast<size_t>(g) * rows + m0 + rr] = stile[g * CQ_ROWS + rr];
                zero[static_cast<size_t>(g) * rows + m0 + rr] = stile[(ng + g) * CQ_ROWS + rr];
            }
        }
    }
}

// ------------------------------------------------------------------------------------------- stored form
// Codes (one byte each) -> the three nibble-packed arrays and byte zero-points of the stored form, in one launch.
// Eight codes c0..c7 become one word with nibble order c0 c2 c4 c6 c1 c3 c5 c7.
__device__ __forceinline__ uint32_t pack8(uint32_t a, uint32_t b) {     // a = c0..c3, b = c4..c7, one byte each
    // even codes c0 c2 c4 c6 to the low half, odd ones to the high half, then adjacent nibbles together
    const uint32_t even = __byte_perm(a, b, 0x6420) & 0x0F0F0F0Fu, odd = __byte_perm(a, b, 0x7531) & 0x0F0F0F0Fu;
    const uint32_t e = even | (even >> 4), o = odd | (odd >> 4);        // byte 0: c0 c2, byte 2: c4 c6
    return __byte_perm(e, o, 0x6420);
}

// 11008 x 4096, r = 512 (23 MB in and out): 4.9 us; five launches with a strided byte gather took about 40.
constexpr int PK_THREADS = 256;
constexpr int PK_K = 64, PK_N = 128;       // a tile of V: 64 ranks x 128 columns

struct PackParams {
    const uint8_t* uc;         // (M, r)
    const uint8_t* vc;         // (r, N)
    const uint16_t* uzb;       // (M, ng) bfloat16
    const uint16_t* vzb;       // (ng, N) bfloat16
    uint32_t* uq;              // (M, r / 8) words
    uint32_t* vq;              // (N, r / 8)
    uint32_t* vt;              // (r, N / 8)
    uint8_t* uz;
    uint8_t* vz;
    int M, N, r;
    int u_blocks, v_blocks, z_blocks;
    int vec;                   // uc and vc are 16-byte aligned
};

// eight consecutive codes (p is a multiple of 8 behind an array that `vec` says is aligned)
__device__ __forceinline__ uint2 load8(const uint8_t* p, int vec) {
    if (vec) return __ldg(reinterpret_cast<const uint2*>(p));
    uint2 v = make_uint2(0, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v.x |= static_cast<uint32_t>(p[i]) << (8 * i);
        v.y |= static_cast<uint32_t>(p[4 + i]) << (8 * i);
    }
    return v;
}

// Blocks [0, u_blocks): U, two words per thread and step.  Then v_blocks tiles of V: read once, written in both orders (the
// transposing gather goes through shared memory; one byte per load and a different row per lane took ten times as long).
// Then z_blocks for the zero-points.
__global__ void __launch_bounds__(PK_THREADS) pack_delta_kernel(const PackParams p) {
    __shared__ uint8_t tile[PK_K][PK_N + 4];
    int b = blockIdx.x;
    if (b < p.u_blocks) {
        const size_t words = static_cast<size_t>(p.M) * (p.r >> 3);
        for (size_t i = static_cast<size_t>(b) * PK_THREADS + threadIdx.x; i < words; i += static_cast<size_t>(p.u_blocks) * PK_THREADS) {
            const uint2 c = load8(p.uc + i * 8, p.vec);
            p.uq[i] = pack8(c.x, c.y);
        }
        return;
    }
    b -= p.u_blocks;
    if (b < p.v_blocks) {
        const int nt = (p.N + PK_N - 1) / PK_N;
        const int k0 = b / nt * PK_K, n0 = (b - b / nt * nt) * PK_N;
        // in: a thread takes eight codes of one rank; they are one word of vt
        for (int e = threadIdx.x; e < PK_K * PK_N / 8; e += PK_THREADS) {
            const int k = e / (PK_N / 8), n = e % (PK_N / 8) * 8;
            if (n0 + n < p.N) {                                           // N is a multiple of 8
                const size_t at = static_cast<size_t>(k0 + k) * p.N + n0 + n;
                const uint2 c = load8(p.vc + at, p.vec);
                p.vt[at >> 3] = pack8(c.x, c.y);
                *reinterpret_cast<uint32_t*>(&tile[k][n]) = c.x;
                *reinterpret_cast<uint32_t*>(&tile[k][n + 4]) = c.y;
            }
        }
        __syncthreads();
        // out: eight ranks of one column are one word of vq; eight threads cover the 32 bytes of a column
        for (int e = threadIdx.x; e < PK_K * PK_N / 8; e += PK_THREADS) {
            const int n = e / (PK_K / 8), k = e % (PK_K / 8) * 8;
            if (n0 + n < p.N) {
                uint32_t c[2] = {0, 0};
#pragma unroll
                for (int i = 0; i < 8; ++i) c[i >> 2] |= static_cast<uint32_t>(tile[k + i][n]) << (8 * (i & 3));
                p.vq[static_cast<size_t>(n0 + n) * (p.r >> 3) + ((k0 + k) >> 3)] = pack8(c[0], c[1]);
            }
        }
        return;
    }
    b -= p.v_blocks;
    const int ng = p.r >> 7;
    const size_t nu = static_cast<size_t>(p.M) * ng, total = nu + static_cast<size_t>(p.N) * ng;
    for (size_t i = static_cast<size_t>(b) * PK_THREADS + threadIdx.x; i < total; i += static_cast<size_t>(p.z_blocks) * PK_THREADS) {
        const bool is_u = i < nu;
        const size_t e = is_u ? i : i - nu;
        const uint16_t z = (is_u ? p.uzb : p.vzb)[e];
        (is_u ? p.uz : p.vz)[e] = static_cast<uint8_t>(static_cast<int>(__uint_as_float(static_cast<uint32_t>(z) << 16)));
    }
}

}  // namespace ade
