// FP32 triangular solve of up to 32 right-hand sides (a strip) by one or more warps, shared by
// the grouped strsm plans (grouped.cu) and the inversion of the blocked trsm's
// diagonal blocks (trsm.cu).
//
// The triangle is cut into 32-row blocks, dealt round robin to the strip's W warps.  For block
// i a warp adds op(A)[i, l] X_l of every earlier block to a register tile (packed FP32 FMAs, 8
// rows of 4 columns per lane), takes the whole sum from B at once, and solves the 32 x 32
// diagonal block one column per lane, every row of a column in one thread, so no pivot is
// broadcast between lanes.  X_i stays in shared memory for the blocks after it; with more than
// one warp an mbarrier per block says that it is there.  Taking the sum at once is for
// accuracy: against a dominant diagonal the products are small beside B, and subtracting them
// one by one would round at B's size each time (measured: 9.6e-7 of the largest entry at order
// 255).  An upper triangle is solved as the lower one that reversing rows and columns gives
// (negative strides), and a transposed one by the strides alone, so there is one instance of
// the arithmetic.
//
// Bound: shared-memory reads for a batch (twelve wavefronts per step of a tile), the chain
// last tile -> diagonal block (about 1440 + 860 cycles) for a lone large problem.  Two or four
// warps per strip keep the chain covered: while one solves a block, the others sum the
// earlier tiles of the next ones.  One warp per block, each waiting for its turn, held the
// registers and ring slots of eight warps for the work of four: 0.102 ms against 0.077 for
// 2048 problems of order 8..256.  Each warp streams its tiles through a private ring of two
// slots with cp.async, so copies need no barrier.
#pragma once

#include "mbg_internal.cuh"
#include "gemm_f32_tile.cuh"
#include "tc_ptx.cuh"

namespace mbg {
namespace ws {

constexpr int RB = 32;              // rows per block, right-hand sides per group
constexpr int SLOT = RB * RB;       // floats per ring slot: one tile


// A tile's element (r, l) sits at l * 32 + (r ^ 4 (l % 8)): its columns contiguous in
// 16-byte chunks that are permuted by column, so that copies along either dimension,
// column reads by one thread and broadcasts are free of bank conflicts.
__device__ __forceinline__ int at(int r, int l) { return l * RB + (r ^ ((l & 7) << 2)); }

__device__ __forceinline__ void copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}

// Starts the copy of a rows x cols tile, element (r, l) at p[r * sr + l * sl] (one of the
// strides is 1 or -1).  Elements outside are left as they are: they only ever enter rows
// and columns that are not part of the problem.  vec: 16-byte copies (sr 1, p and sl
// 16-byte aligned).
__device__ __forceinline__ void copy_tile(float* dst, const float* p, i64 sr, i64 sl, int rows, int cols, bool vec,
                                          int lane) {
    asm volatile("" : "+l"(sr), "+l"(sl));  // or their multiples are kept (and spilled) between copies
    if (vec) {
        const int r = 4 * (lane & 7), n = min(4, rows - r);
        const float* q = p + r + (lane >> 3) * sl;
        if (n > 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += 4 * sl) {
                const int l = 4 * j + (lane >> 3);
                if (l < cols) copy16(dst + at(r, l), q, 4 * n);
            }
        }
    } else if (sr == 1 || sr == -1) {  // lanes along the rows
        if (lane < rows) {
            const float* q = p + lane * sr;
#pragma unroll 8
            for (int l = 0; l < cols; ++l, q += sl) copy4(dst + at(lane, l), q);
        }
    } else {  // eight columns (contiguous) of four rows per copy
        const int l0 = lane & 7, r0 = lane >> 3;
#pragma unroll
        for (int j = 0; j < RB / 8; ++j) {
            const int l = l0 + 8 * j;
            if (l < cols) {
                const float* q = p + r0 * sr + l * sl;
#pragma unroll
                for (int i = 0; i < RB / 4; ++i, q += 4 * sr)
                    if (r0 + 4 * i < rows) copy4(dst + at(r0 + 4 * i, l), q);
            }
        }
    }
}

struct Problem {
    const float* a;  // op(A)[0, 0] in solve order, element (r, l) at a[r * sr + l * sl]
    i64 sr, sl;
    float* b;        // B[0, first column] in solve order, element (r, c) at b[r * sb + c * ldb], sb = 1 or -1
    i64 sb, ldb;
    int n, cols;     // order, right-hand sides (at most 32)
    float alpha;
    bool unit;
};

// op(A) of order n at `a` (column-major, lda) in solve order.
__device__ __forceinline__ void solve_order(Problem& p, const float* a, i64 lda, int n, bool lower, bool trans) {
    const i64 sr = trans ? lda : 1, sl = trans ? 1 : lda;
    p.a = lower ? a : a + (n - 1) * (lda + 1);
    p.sr = lower ? sr : -sr;
    p.sl = lower ? sl : -sl;
    p.n = n;
}

// y += a * b where `on`: predicated, so that a column's loads can be issued before its pivot
// is known to be nonzero.
__device__ __forceinline__ void fma_if(unsigned long long& y, unsigned long long a, unsigned long long b, int on) {
    asm("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p fma.rn.f32x2 %0, %1, %2, %0; }" : "+l"(y) : "l"(a), "l"(b), "r"(on));
}
__device__ __forceinline__ void fma_if(float& y, float a, float b, int on) {
    asm("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p fma.rn.f32 %0, %1, %2, %0; }" : "+f"(y) : "f"(a), "f"(b), "r"(on));
}

// acc += T X for one tile, X as [l][column]: lane (rg, cg) = (lane % 4, lane / 4) holds rows
// 8 rg .. 8 rg + 7 of columns 4 cg .. 4 cg + 3, so a step of l reads three 16-byte words for
// 32 multiply-adds.  SKIP leaves out the products with a zero of X.  (One column per lane with all 32 rows reads nine, each of T's a
// broadcast that still takes two wavefronts.)
template <bool SKIP>
__device__ __forceinline__ void tile_update(unsigned long long (&acc)[4][4], const float* tile, const float* x,
                                            int lane) {
    const int r = 8 * (lane & 3), c = 4 * (lane >> 2);
#pragma unroll 1
    for (int l0 = 0; l0 < RB; l0 += 16) {
#pragma unroll SKIP ? 4 : 16
        for (int j = 0; j < 16; ++j) {
            const int sw = 4 * (j & 7);
            const float4 v = *reinterpret_cast<const float4*>(x + (l0 + j) * RB + c);
            const ulonglong2 t0 = *reinterpret_cast<const ulonglong2*>(tile + (l0 + j) * RB + (r ^ sw));
            const ulonglong2 t1 = *reinterpret_cast<const ulonglong2*>(tile + (l0 + j) * RB + ((r + 4) ^ sw));
            const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned long long vv = f32t::f2_pack(vs[k], vs[k]);
                if constexpr (SKIP) {
                    const int on = vs[k] != 0.0f;
                    fma_if(acc[k][0], t0.x, vv, on);
                    fma_if(acc[k][1], t0.y, vv, on);
                    fma_if(acc[k][2], t1.x, vv, on);
                    fma_if(acc[k][3], t1.y, vv, on);
                } else {
                    f32t::f2_fma(acc[k][0], t0.x, vv);
                    f32t::f2_fma(acc[k][1], t0.y, vv);
                    f32t::f2_fma(acc[k][2], t1.x, vv);
                    f32t::f2_fma(acc[k][3], t1.y, vv);
                }
            }
        }
    }
}

// One column per thread: y := D^-1 y for the 32 x 32 diagonal block D, whose diagonal holds the
// negated reciprocals; straight-line code, so that the loads of later columns are issued
// ahead of the chain of pivots.  SKIP leaves a column alone where its pivot is zero
// (src/level3/trsm.mojo:130-148), which takes 1670 cycles for a warp alone against 860 without
// (a predicate per multiply-add).  The result differs only where a zero pivot meets an
// infinity or a NaN, so the caller runs SKIP only if the other found a zero: the value
// returned says that no pivot was zero.
// SKIP's loads are volatile, or the compiler keeps the other's (the whole block) for it, in
// local memory.
template <bool VOLATILE>
__device__ __forceinline__ ulonglong2 load_pairs(const float* p) {
    if constexpr (!VOLATILE) return *reinterpret_cast<const ulonglong2*>(p);
    ulonglong2 v;
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                 : "=l"(v.x), "=l"(v.y)
                 : "r"((unsigned)__cvta_generic_to_shared(p)));
    return v;
}
template <bool VOLATILE>
__device__ __forceinline__ float load_one(const float* p) {
    if constexpr (!VOLATILE) return *p;
    return *reinterpret_cast<const volatile float*>(p);
}
template <bool SKIP>
__device__ __forceinline__ bool substitute(unsigned long long (&y)[RB / 2], const float* diag) {
    bool ok = true;
#pragma unroll
    for (int l = 0; l < RB; ++l) {
        const float s = load_one<SKIP>(diag + at(l, l));
        float lo, hi;
        f32t::f2_unpack(y[l / 2], lo, hi);
        const float v = l % 2 ? hi : lo;
        const int live = v != 0.0f;
        ok = ok && live;
        const float nv = v * s;  // -x
        if (l % 2) {
            hi = SKIP && !live ? v : -nv;
        } else {
            if constexpr (SKIP) fma_if(hi, load_one<SKIP>(diag + at(l + 1, l)), nv, live);
            else hi = fmaf(diag[at(l + 1, l)], nv, hi);
            lo = SKIP && !live ? v : -nv;
        }
        y[l / 2] = f32t::f2_pack(lo, hi);
        const unsigned long long nn = f32t::f2_pack(nv, nv);
#pragma unroll
        for (int q = (l / 2 + 1) / 2; q < RB / 4; ++q) {
            const ulonglong2 t = load_pairs<SKIP>(diag + at(4 * q, l));
            if constexpr (SKIP) {
                if (2 * q > l / 2) fma_if(y[2 * q], t.x, nn, live);
                fma_if(y[2 * q + 1], t.y, nn, live);
            } else {
                if (2 * q > l / 2) f32t::f2_fma(y[2 * q], t.x, nn);
                f32t::f2_fma(y[2 * q + 1], t.y, nn);
            }
        }
    }
    return ok;
}

// One warp's part of a strip: blocks wi, wi + W, ... of nblk = ceil(n / 32).  X: the strip's nblk
// slots; ring: this warp's two slots; bars: an mbarrier of count 1 per block, initialised
// (unused when W is 1); zeros: an int per block, set where X has a zero, whose products are left
// out (unused for an identity).  IDENT: the right-hand sides are the first columns of the
// identity, B is only written.
template <bool IDENT>
__device__ __forceinline__ void solve_strip(const Problem& p, int wi, int W, float* X, float* ring, uint64_t* bars,
                                            volatile int* zeros, int lane, int* err) {
    const int nblk = (p.n + RB - 1) / RB;
    const bool va = p.sr == 1 && p.sl % 4 == 0 && reinterpret_cast<uintptr_t>(p.a) % 16 == 0;
    const bool vb = p.sb == 1 && p.ldb % 4 == 0 && reinterpret_cast<uintptr_t>(p.b) % 16 == 0;
    // the warp's tiles in the order of their use, (i, 0) .. (i, i) for each of its blocks i,
    // through alternating slots; a block of B goes with its row's first tile
    int fi = wi, fl = 0, fslot = 0;
    auto fetch = [&] {
        if (fi < nblk) {
            const int rows = min(RB, p.n - RB * fi);
            if (!IDENT && fl == 0) copy_tile(X + fi * SLOT, p.b + RB * fi * p.sb, p.sb, p.ldb, rows, p.cols, vb, lane);
            copy_tile(ring + fslot * SLOT, p.a + RB * (fi * p.sr + fl * p.sl), p.sr, p.sl, rows, fl == fi ? rows : RB, va,
                      lane);
            if (fl++ == fi) {
                fi += W;
                fl = 0;
            }
        }
        f32t::cpa_commit();
        fslot ^= 1;
    };
    fetch();
    fetch();
    int slot = 0;
    for (int i = wi; i < nblk; i += W) {
        const int rows = min(RB, p.n - RB * i);
        float* const Xi = X + i * SLOT;
        unsigned long long acc[4][4];
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e / 4][e % 4] = 0ULL;
        auto reciprocals = [&](float* diag) {
            __syncwarp();
            diag[at(lane, lane)] = p.unit ? -1.0f : -1.0f / diag[at(lane, lane)];
        };
        for (int l = 0; l < i; ++l) {
            if (l + 1 < i) {
                f32t::cpa_wait<1>();
            } else {  // the diagonal block's reciprocals, in the shadow of the wait for X_l
                f32t::cpa_wait<0>();
                reciprocals(ring + (slot ^ 1) * SLOT);
            }
            if (W > 1 && !tc::mbar_wait(bars + l, 0, err, 41)) {
                f32t::cpa_wait<0>();
                return;
            }
            __syncwarp();  // the whole of the tile has landed
            if (!IDENT && zeros[l]) tile_update<true>(acc, ring + slot * SLOT, X + l * SLOT, lane);
            else tile_update<false>(acc, ring + slot * SLOT, X + l * SLOT, lane);
            __syncwarp();
            fetch();
            slot ^= 1;
        }
        float* const diag = ring + slot * SLOT;
        f32t::cpa_wait<1>();
        if (i == 0) reciprocals(diag);
        __syncwarp();
        if (IDENT || i > 0) {  // the right-hand sides less the sums, from here one column per lane
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = 8 * (lane & 3) + 4 * h, c = 4 * (lane >> 2) + k;
                    float4* const q = reinterpret_cast<float4*>(Xi + at(r, c));
                    float4 v, s;
                    if constexpr (IDENT) {
                        const int d = i == 0 ? c - r : -1;
                        v = make_float4(d == 0, d == 1, d == 2, d == 3);
                    } else {
                        v = *q;
                        v = make_float4(p.alpha * v.x, p.alpha * v.y, p.alpha * v.z, p.alpha * v.w);
                    }
                    f32t::f2_unpack(acc[k][2 * h], s.x, s.y);
                    f32t::f2_unpack(acc[k][2 * h + 1], s.z, s.w);
                    *q = make_float4(v.x - s.x, v.y - s.y, v.z - s.z, v.w - s.w);
                }
            __syncwarp();
        }
        unsigned long long y[RB / 2];
        auto load = [&] {
            const float scale = IDENT || i > 0 ? 1.0f : p.alpha;
#pragma unroll
            for (int q = 0; q < RB / 4; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(Xi + at(4 * q, lane));
                y[2 * q] = f32t::f2_pack(scale * v.x, scale * v.y);
                y[2 * q + 1] = f32t::f2_pack(scale * v.z, scale * v.w);
            }
        };
        load();
        if (rows < RB) {  // rows past the end reach no row of the problem; a zero there is no pivot
#pragma unroll
            for (int e = 0; e < RB / 2; ++e) {
                float lo, hi;
                f32t::f2_unpack(y[e], lo, hi);
                y[e] = f32t::f2_pack(2 * e < rows ? lo : 1.0f, 2 * e + 1 < rows ? hi : 1.0f);
            }
        }
        // (the first block of an identity has zero pivots in every column but one)
        const bool skip = (IDENT && i == 0) || __any_sync(0xffffffffu, !substitute<false>(y, diag) && lane < p.cols);
        if (skip) {
            asm volatile("" ::: "memory");  // D and the columns are read again, not kept in registers
            load();
            substitute<true>(y, diag);
        }
        __syncwarp();  // every lane has read its column and the diagonal block
        if (i + 1 < nblk) {  // `rows` is 32 here
#pragma unroll
            for (int l = 0; l < RB; l += 2) {
                float lo, hi;
                f32t::f2_unpack(y[l / 2], lo, hi);
                Xi[l * RB + lane] = lo;
                Xi[(l + 1) * RB + lane] = hi;
            }
            if (!IDENT && lane == 0) zeros[i] = skip;
            if (W > 1) {
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(bars + i);
            }
        }
#pragma unroll
        for (int q = 0; q < RB / 4; ++q)  // the diagonal block's slot takes the columns for the store
            *reinterpret_cast<ulonglong2*>(diag + at(4 * q, lane)) = make_ulonglong2(y[2 * q], y[2 * q + 1]);
        __syncwarp();
        float* const brow = p.b + RB * i * p.sb;
        if (vb && rows == RB) {
            const int r = 4 * (lane & 7);
            float* q = brow + r + (lane >> 3) * p.ldb;
#pragma unroll
            for (int j = 0; j < 8; ++j, q += 4 * p.ldb) {
                const int c = 4 * j + (lane >> 3);
                if (c < p.cols) *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(diag + at(r, c));
            }
        } else if (lane < rows) {
            float* q = brow + lane * p.sb;
#pragma unroll 8
            for (int c = 0; c < p.cols; ++c, q += p.ldb) *q = diag[at(lane, c)];
        }
        __syncwarp();
        fetch();
        slot ^= 1;
    }
    f32t::cpa_wait<0>();
}

}  // namespace ws
}  // namespace mbg
