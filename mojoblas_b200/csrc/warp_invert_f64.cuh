// FP64 inverse of a triangle's diagonal block, 32 columns (a strip) at a time: the strip solve of
// warp_solve.cuh on identity columns, with its tiles on the FP64 tensor pipe.
//
// The block is cut into 32-row blocks, dealt round robin to the strip's W warps.  For block i a
// warp adds op(A)[i, l] X_l of every earlier block (mma.sync m8n8k4, a 32 x 32 tile per step),
// takes the sum from the identity at once, and solves the 32 x 32 diagonal block one column per
// lane; X_i stays in shared memory for the blocks after it, and an mbarrier per block says that
// it is there.  An upper triangle is solved as the lower one that reversing rows and columns
// gives, a transposed one by the strides alone.
//
// Bound: the FP64 pipe (2048 cycles of a scheduler for a tile) for the first strips, the chain last
// tile -> diagonal block for the others.
#pragma once

#include "mbg_internal.cuh"
#include "tc_ptx.cuh"

namespace mbg {
namespace wd {

constexpr int RB = 32;          // rows per block, columns per strip
constexpr int SLOT = RB * RB;   // doubles per slot: one tile

// A tile's element (r, l) sits at l * 32 + (r ^ 4 (l % 8)): copies, column reads and the fragments
// of the tensor pipe (four consecutive l of four consecutive r per half warp) hit distinct banks.
__device__ __forceinline__ int at(int r, int l) { return l * RB + (r ^ ((l & 7) << 2)); }

__device__ __forceinline__ void copy8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy16(double* dst, const double* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Starts the copy of a rows x cols tile, element (r, l) at p[r * sr + l * sl] (one of the strides is
// 1 or -1); what lies outside is left as it is and only ever enters rows outside the problem.
// vec: 16-byte copies (sr 1, p and sl 16-byte aligned).
__device__ __forceinline__ void copy_tile(double* dst, const double* p, i64 sr, i64 sl, int rows, int cols, bool vec,
                                          int lane) {
    if (vec) {
        const int r = 2 * (lane & 15), n = min(2, rows - r);
        const double* q = p + r + (lane >> 4) * sl;
        if (n > 0) {
#pragma unroll 8
            for (int l = lane >> 4; l < cols; l += 2, q += 2 * sl) copy16(dst + at(r, l), q, 8 * n);
        }
    } else if (sr == 1 || sr == -1) {  // lanes along the rows
        if (lane < rows) {
            const double* q = p + lane * sr;
#pragma unroll 8
            for (int l = 0; l < cols; ++l, q += sl) copy8(dst + at(lane, l), q);
        }
    } else {  // lanes along the (contiguous) columns
        if (lane < cols) {
            const double* q = p + lane * sl;
#pragma unroll 8
            for (int r = 0; r < rows; ++r, q += sr) copy8(dst + at(r, lane), q);
        }
    }
}

// acc += T X for one tile, X's element (l, c) at at(c, l): fragment (i, j) holds row 8 i + lane / 4,
// columns 8 j + 2 (lane % 4) + {0, 1}.
__device__ __forceinline__ void tile_update(double (&acc)[4][4][2], const double* tile, const double* x, int lane) {
    const int lr = lane >> 2, lk = lane & 3;
#pragma unroll 2
    for (int k0 = 0; k0 < RB; k0 += 4) {
        const int l = k0 + lk;
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = tile[at(8 * i + lr, l)];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = x[at(8 * j + lr, l)];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                             : "+d"(acc[i][j][0]), "+d"(acc[i][j][1])
                             : "d"(a[i]), "d"(b[j]));
    }
}

// One column per thread: y := D^-1 y for the 32 x 32 diagonal block D, whose diagonal holds the
// negated reciprocals.  SKIP leaves a column alone where its pivot is zero
// (src/level3/trsm.mojo:130-148); its loads are volatile, or the compiler keeps the other's for it.
template <bool SKIP>
__device__ __forceinline__ double load(const double* p) {
    if constexpr (SKIP) return *reinterpret_cast<const volatile double*>(p);
    return *p;
}
template <bool SKIP>
__device__ __forceinline__ bool substitute(double (&y)[RB], const double* diag) {
    bool ok = true;
#pragma unroll
    for (int l = 0; l < RB; ++l) {
        const bool live = y[l] != 0.0;
        ok = ok && live;
        const double nv = y[l] * load<SKIP>(diag + at(l, l));  // -x
        if (!SKIP || live) {
            y[l] = -nv;
#pragma unroll
            for (int r = l + 1; r < RB; ++r) y[r] = fma(load<SKIP>(diag + at(r, l)), nv, y[r]);
        }
    }
    return ok;
}

struct Strip {
    const double* a;  // op(A) from the strip's first row and column on, in solve order: (r, l) at a[r * sr + l * sl]
    i64 sr, sl;
    double* w;        // the inverse there, (r, c) at w[r * sw + c * ldw], sw = 1 or -1
    i64 sw, ldw;
    int n, cols;      // rows (and columns of op(A)) from there on; columns of the strip (at most 32)
    bool unit;
};

// One warp's part of a strip: blocks wi, wi + W, ... of ceil(n / 32).  X: a slot per block; ring:
// this warp's two slots; bars: an mbarrier of count 1 per block, initialised.
__device__ __forceinline__ void invert_strip(const Strip& p, int wi, int W, double* X, double* ring, uint64_t* bars,
                                             int lane, int* err) {
    const int nblk = (p.n + RB - 1) / RB;
    const bool vec = p.sr == 1 && p.sl % 2 == 0 && reinterpret_cast<uintptr_t>(p.a) % 16 == 0;
    int fi = wi, fl = 0, fslot = 0;
    auto fetch = [&] {  // the next tile of (i, 0) .. (i, i), i = wi, wi + W, ..., into the other slot
        if (fi < nblk) {
            const int rows = min(RB, p.n - RB * fi);
            copy_tile(ring + fslot * SLOT, p.a + RB * (fi * p.sr + fl * p.sl), p.sr, p.sl, rows, fl == fi ? rows : RB, vec,
                      lane);
            if (fl++ == fi) {
                fi += W;
                fl = 0;
            }
        }
        commit();
        fslot ^= 1;
    };
    fetch();
    fetch();
    int slot = 0;
    for (int i = wi; i < nblk; i += W) {
        const int rows = min(RB, p.n - RB * i);
        double* const Xi = X + i * SLOT;
        auto reciprocals = [&](double* d) {
            __syncwarp();
            d[at(lane, lane)] = p.unit ? -1.0 : -1.0 / d[at(lane, lane)];
        };
        double y[RB];
        {
            double acc[4][4][2];
#pragma unroll
            for (int e = 0; e < 32; ++e) acc[e / 8][e / 2 % 4][e % 2] = 0.0;
            for (int l = 0; l < i; ++l) {
                if (l + 1 < i) {
                    wait<1>();
                } else {  // the diagonal block's reciprocals, in the shadow of the wait for X_l
                    wait<0>();
                    reciprocals(ring + (slot ^ 1) * SLOT);
                }
                if (!tc::mbar_wait(bars + l, 0, err, 42)) {
                    wait<0>();
                    return;
                }
                __syncwarp();  // the whole of the tile has landed
                tile_update(acc, ring + slot * SLOT, X + l * SLOT, lane);
                __syncwarp();
                fetch();
                slot ^= 1;
            }
            wait<1>();
            if (i == 0) reciprocals(ring + slot * SLOT);
            // the identity less the sum, then one column per lane
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int row = 8 * r + (lane >> 2), col = 8 * c + 2 * (lane & 3) + e;
                        Xi[at(row, col)] = (i == 0 && row == col ? 1.0 : 0.0) - acc[r][c][e];
                    }
            __syncwarp();
        }
        double* const diag = ring + slot * SLOT;
        auto column = [&] {
#pragma unroll
            for (int r = 0; r < RB; ++r) y[r] = r < rows ? Xi[at(r, lane)] : 1.0;  // rows past the end reach no other
        };
        column();
        // (the first block of an identity has zero pivots in every column but one)
        const bool skip = i == 0 || __any_sync(0xffffffffu, !substitute<false>(y, diag) && lane < p.cols);
        if (skip) {
            column();
            substitute<true>(y, diag);
        }
        __syncwarp();  // every lane has read its column and the diagonal block
        if (i + 1 < nblk) {  // `rows` is 32 here
#pragma unroll
            for (int l = 0; l < RB; ++l) Xi[at(lane, l)] = y[l];
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bars + i);
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) diag[at(r, lane)] = y[r];
        __syncwarp();
        if (lane < rows) {
            double* q = p.w + (RB * i + lane) * p.sw;
#pragma unroll 8
            for (int c = 0; c < p.cols; ++c, q += p.ldw) *q = diag[at(lane, c)];
        }
        __syncwarp();
        fetch();
        slot ^= 1;
    }
    wait<0>();
}

}  // namespace wd
}  // namespace mbg
