// Grouped split-precision sgemm (BF16x3 / BF16x6) on the tensor cores: thousands of
// independent problems of uneven sizes in one persistent tcgen05 launch.
//
// The reference has no batched interface (a mojoBLAS caller loops over gemm,
// src/level3/gemm.mojo:56).  The single-call split kernel (tc_gemm.cu) runs a
// pre-pass that writes bf16 planes and then TMA-loads them; for problems of 16 to
// 512 rows that pre-pass would cost more than the products, and TMA needs
// 16-byte-aligned leading dimensions that batched callers rarely have.  Here the
// split is fused into the kernel's producer warps:
//   warps 0..15  producers, two groups of eight that take the 32-deep k slabs in turn, so
//                that one group's loads are in flight while the other splits; in a group
//                four warps per operand, 32 rows of its tile each.  A warp loads its
//                32 x 32 values straight into registers, coalesced along whichever
//                dimension the operand stores contiguously: along the rows a lane holds
//                one row, along k a lane holds one pair of k of sixteen rows.  Either way
//                its values are sixteen k-adjacent pairs, which it splits into TERMS bf16 terms
//                (x1 = bf16(x), x2 = bf16(x - x1), x3 = bf16(x - x1 - x2); each
//                difference is exact) and stores in the tcgen05 K-major layout with the
//                64-byte swizzle, rows and k past the problem's edge as zeros.
//                Then a proxy fence and an arrival on the stage's "full" barrier;
//   warp 16      lane 0 issues the TERMS (TERMS + 1) / 2 products per 16-deep k
//                step into a TMEM accumulator of 128 x BN fp32 (BN = 64 or 128
//                per problem), restarted every 128 k (the tensor core's fp32
//                accumulation truncates) into the other of two buffers;
//   warps 17..19 prefetch the slabs six (BF16x3: eight) ahead of the products into L2: a producer's
//                registers hold one slab of loads, too little in flight to cover HBM;
//   warps 20..27 epilogue: add each 128-k chunk into fp32 registers with
//                round-to-nearest, then alpha / beta and the column-major store;
//                the other TMEM buffer lets the next tile's products run meanwhile.
// Registers are dealt by role (setmaxnreg).  Tiles (128 rows, BN columns of one problem; one
// descriptor each, read a tile ahead) are ordered by reduction length, longest first, and
// dealt round robin to one persistent CTA per SM.  All waits are bounded (2 s) and report
// through the library's error flag.
//
// Bound: shared memory, which carries per 32-deep slab of a 128 x 128 tile the products' operand
// reads (60 KB with A from the collector), the terms' stores (48 KB) and the loads' lines
// (40 KB), and the start and end of tiles of five slabs on average.  4096 problems (m, n, k
// log-uniform 16..512, NN, BF16x6): 0.534 ms (0.567 without the prefetch), of which 0.36 ms remain
// without loads, splits and stores of C.  Copying each slab to shared memory first (4-byte cp.async,
// one slab ahead) and splitting from there took 0.697 ms: about 50 cycles for each copy instruction of
// eight producer warps, and branches around each column of the epilogue's stores.  For many small
// aligned problems, which HBM bounds, the prefetch is what makes up for its 16-byte copies: 3000 of
// 96 x 96 x 96, TN, BF16x3 94 us with them, 148 with neither and 91 with the prefetch and the loads of
// aligned pairs.
#include "mbg_internal.cuh"
#include "gemm_f32_tile.cuh"
#include "schedule.cuh"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <vector>

namespace mbg {
namespace gtc {

using namespace tc;

constexpr int GBN = 128;       // widest tile (TMEM buffer stride)
constexpr int GBKB = 64;       // k slab: 32 bf16 per row, 64-byte swizzle
constexpr int GBK = 32;
constexpr int GCHUNK = 4;      // slabs per TMEM accumulation chunk
constexpr int GGROUPS = 2;                // producer groups, taking slabs in turn
constexpr int GGROUP_WARPS = 8;           // 4 for op(A), 4 for op(B)^T
constexpr int GPROD_WARPS = GGROUPS * GGROUP_WARPS;
constexpr int GMMA_WARP = GPROD_WARPS;
constexpr int GPREFETCH_WARPS = 3;        // with the MMA warp: registers are dealt per four warps
constexpr int GEPI_WARP0 = GMMA_WARP + 4;
constexpr int GEPI_WARPS = 8;
constexpr int GTHREADS = 32 * (GEPI_WARP0 + GEPI_WARPS);
// 896 threads start with 72 registers: 64512 = 512 x 72 (producers) + 128 x 24 + 256 x 96 (epilogue)
constexpr int GREGS_PROD = 72, GREGS_MMA = 24, GREGS_EPI = 96;
static_assert(32 * GPROD_WARPS * GREGS_PROD + 128 * GREGS_MMA + 32 * GEPI_WARPS * GREGS_EPI <= GTHREADS * 72,
              "the register split must fit what the CTA was launched with");

template <int TERMS>
struct GCfg {
    static constexpr int A_PLANE = BM * GBKB;   // 8 KB
    static constexpr int B_PLANE = GBN * GBKB;  // 8 KB
    static constexpr int STAGE_BYTES = TERMS * (A_PLANE + B_PLANE);
    static constexpr int STAGES = TERMS == 3 ? 4 : 6;  // split planes in flight to the MMA warp
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
    static constexpr int NPROD = TERMS * (TERMS + 1) / 2;
    static constexpr int AHEAD = TERMS == 3 ? 6 : 8;  // slabs prefetched ahead of the products
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

// One tile of one problem.  Row i of op(A) (column j of op(B)) within the tile, k index l, sits at
// a[i * lda + l] (a_kcontig) or a[i + l * lda]; likewise b.
struct __align__(16) TcTile {
    const float* a;  // the tile's first row
    const float* b;  // the tile's first column
    float* c;        // the tile's corner
    i64 lda, ldb, ldc;
    int nkb, last;   // k slabs (0 when alpha == 0 or k == 0: C := beta C only), elements of the last
    int rows, cols;  // of the tile inside the problem
    int bn;          // tile columns: 64 or 128
    int kcontig;     // bit 0: op(A)'s k is the contiguous dimension, bit 1: op(B)'s; bits 2, 3: and a pair of k is
                     // 8-byte aligned in every row
    float alpha, beta;
};

// A warp's 32 rows (rw0 ..) of a k slab, `left` deep from p on, as 16 k-adjacent pairs per lane: pair i
// is k (2 i, 2 i + 1) of row rw0 + lane, or, KC (k contiguous), k (2 q, 2 q + 1) of row
// rw0 + 2 i + h with (h, q) = (lane / 16, lane % 16), so that a load covers two rows of 128 bytes.
// Zeros past the operand's rows and past the slab's end.  even: pairs are 8-byte aligned.
template <bool KC>
__device__ __forceinline__ void load_pairs(float (&v)[32], const float* __restrict__ p, i64 ld, int rw0, int rows,
                                           int left, int lane, bool even = false) {
    if (KC) {
        const int h = lane >> 4, k = 2 * (lane & 15);
        const float* q = p + i64(rw0 + h) * ld + k;
        const bool on0 = k < left, on1 = k + 1 < left;
        if (rw0 + 32 <= rows && left == GBK && even) {
#pragma unroll
            for (int i = 0; i < 16; ++i, q += 2 * ld) {
                const float2 w = __ldg(reinterpret_cast<const float2*>(q));
                v[2 * i] = w.x;
                v[2 * i + 1] = w.y;
            }
        } else if (rw0 + 32 <= rows && left == GBK) {
#pragma unroll
            for (int i = 0; i < 16; ++i, q += 2 * ld) {
                v[2 * i] = __ldg(q);
                v[2 * i + 1] = __ldg(q + 1);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i, q += 2 * ld) {
                const bool r = rw0 + h + 2 * i < rows;
                v[2 * i] = r && on0 ? __ldg(q) : 0.0f;
                v[2 * i + 1] = r && on1 ? __ldg(q + 1) : 0.0f;
            }
        }
    } else {
        const float* q = p + rw0 + lane;
        const bool r = rw0 + lane < rows;
        if (left == GBK) {
#pragma unroll
            for (int l = 0; l < 32; ++l, q += ld) v[l] = r ? __ldg(q) : 0.0f;
        } else {
#pragma unroll
            for (int l = 0; l < 32; ++l, q += ld) v[l] = r && l < left ? __ldg(q) : 0.0f;
        }
    }
}

// The pairs' TERMS bf16 terms, a plane each, at their 64-byte-swizzled places (16-byte chunk c of row
// r sits at c ^ (r / 2) % 4).  A pair is rounded by one bf16x2 conversion, and what its terms
// leave is taken exactly by a packed fma with -1.
template <int TERMS, bool KC>
__device__ __forceinline__ void split_store(const float (&v)[32], uint8_t* plane0, int plane_bytes, int rw0, int lane) {
    constexpr unsigned long long MINUS1 = 0xbf800000bf800000ull;
    if (KC) {
        const int h = lane >> 4, q = lane & 15;
        uint8_t* const base = plane0 + (rw0 + h) * GBKB + (q & 3) * 4;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            unsigned long long x = f32t::f2_pack(v[2 * i], v[2 * i + 1]);
            uint8_t* const d = base + 2 * i * GBKB + (((q >> 2) ^ (i & 3)) << 4);
#pragma unroll
            for (int t = 0; t < TERMS; ++t) {
                float lo, hi;
                f32t::f2_unpack(x, lo, hi);
                const __nv_bfloat162 pr = __floats2bfloat162_rn(lo, hi);
                const uint32_t w = *reinterpret_cast<const uint32_t*>(&pr);
                *reinterpret_cast<uint32_t*>(d + t * plane_bytes) = w;
                if (t + 1 < TERMS)
                    f32t::f2_fma(x, f32t::f2_pack(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), MINUS1);
            }
        }
    } else {
        const int r = rw0 + lane, sw = (r >> 1) & 3;
        uint8_t* const rowp = plane0 + r * GBKB;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t w[TERMS][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                unsigned long long x = f32t::f2_pack(v[8 * c + 2 * i], v[8 * c + 2 * i + 1]);
#pragma unroll
                for (int t = 0; t < TERMS; ++t) {
                    float lo, hi;
                    f32t::f2_unpack(x, lo, hi);
                    const __nv_bfloat162 pr = __floats2bfloat162_rn(lo, hi);
                    w[t][i] = *reinterpret_cast<const uint32_t*>(&pr);
                    if (t + 1 < TERMS)
                        f32t::f2_fma(x, f32t::f2_pack(__uint_as_float(w[t][i] << 16), __uint_as_float(w[t][i] & 0xffff0000u)),
                                     MINUS1);
                }
            }
#pragma unroll
            for (int t = 0; t < TERMS; ++t)
                *reinterpret_cast<uint4*>(rowp + t * plane_bytes + ((c ^ sw) << 4)) =
                    make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
        }
    }
}

// Starts the fetch of a tile's k slab kb into L2, a warp's work: a row or a k per lane.
__device__ __forceinline__ void prefetch_slab(const TcTile* d, int kb, int nkb, int lane) {
    const int left = k_left(nkb, d->last, kb, GBK);
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
        const i64 ld = side ? d->ldb : d->lda;
        const int rows = side ? d->cols : d->rows;
        const float* q = side ? d->b : d->a;
        if ((d->kcontig >> side) & 1) {
            q += i64(kb) * GBK + lane * ld;
#pragma unroll 1
            for (int r = lane; r < rows; r += 32, q += 32 * ld) asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
        } else if (lane < left) {
            q += (i64(kb) * GBK + lane) * ld;
#pragma unroll 1
            for (int r = 0; r < rows; r += 32, q += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
        }
    }
}

__device__ __forceinline__ void st_if(float* p, float v, bool on) {  // no branch per element
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q st.global.f32 [%0], %1; }" ::"l"(p), "f"(v), "r"(int(on))
                 : "memory");
}

template <int TERMS>
__global__ void __launch_bounds__(GTHREADS, 1)
grouped_tc_kernel(const TcTile* __restrict__ tiles, int ntiles, int* err) {
    using C = GCfg<TERMS>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE_BYTES);
    uint64_t* empty = full + C::STAGES;
    uint64_t* tfull = empty + C::STAGES;  // [2]
    uint64_t* tempty = tfull + 2;       // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    volatile int* const slabs_done = reinterpret_cast<volatile int*>(tmem_slot + 1);  // slabs the MMA warp has issued
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        *slabs_done = 0;
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(&full[s], GGROUP_WARPS);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], GEPI_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == GMMA_WARP) {
        tmem_alloc(tmem_slot, 2 * GBN);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < GPROD_WARPS) {
        // ---------------- producers: load, split, store ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GREGS_PROD));
        const int group = warp / GGROUP_WARPS, role = warp % GGROUP_WARPS;
        const bool isA = role < 4;
        const int rw0 = 32 * (role & 3);
        uint8_t* const planes = smem + (isA ? 0 : TERMS * C::A_PLANE);
        const int plane_bytes = isA ? C::A_PLANE : C::B_PLANE;
        int it = 0;  // slabs of this CTA before the current tile
        bool ok = true;
        struct View { const float* p; i64 ld; int nkb, last, rows, used, kc; };
        auto view = [&](int t) {
            View o{};
            if (t < ntiles) {
                const TcTile* d = tiles + t;
                o.p = isA ? d->a : d->b;
                o.ld = isA ? d->lda : d->ldb;
                o.nkb = d->nkb;
                o.last = d->last;
                o.rows = isA ? d->rows : d->cols;
                o.used = isA ? BM : d->bn;
                o.kc = (d->kcontig >> (isA ? 0 : 1)) & 5;
            }
            return o;
        };
        View next = view(blockIdx.x);
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            const View o = next;
            next = view(t + gridDim.x);  // a tile ahead
            const i64 slab = o.kc ? i64(GBK) : GBK * o.ld;  // from one slab's start to the next's
            const float* p = o.p + ((it ^ group) & 1) * slab;
            for (int kb = (it ^ group) & 1; kb < o.nkb; kb += GGROUPS, p += GGROUPS * slab) {
                const int s = (it + kb) % C::STAGES, use = (it + kb) / C::STAGES;
                uint8_t* const plane0 = planes + s * C::STAGE_BYTES;
                if (rw0 < o.rows) {
                    float v[32];
                    const int left = k_left(o.nkb, o.last, kb, GBK);
                    if (o.kc) {
                        load_pairs<true>(v, p, o.ld, rw0, o.rows, left, lane, o.kc & 4);
                        if (!mbar_wait(&empty[s], (use & 1) ^ 1, err, 31)) { ok = false; break; }
                        split_store<TERMS, true>(v, plane0, plane_bytes, rw0, lane);
                    } else {
                        load_pairs<false>(v, p, o.ld, rw0, o.rows, left, lane);
                        if (!mbar_wait(&empty[s], (use & 1) ^ 1, err, 31)) { ok = false; break; }
                        split_store<TERMS, false>(v, plane0, plane_bytes, rw0, lane);
                    }
                } else {
                    if (!mbar_wait(&empty[s], (use & 1) ^ 1, err, 31)) { ok = false; break; }
                    if (rw0 < o.used) {  // padding rows: zero terms
#pragma unroll
                        for (int tt = 0; tt < TERMS; ++tt)
#pragma unroll
                            for (int c = 0; c < 4; ++c)
                                *reinterpret_cast<uint4*>(plane0 + tt * plane_bytes + (rw0 + lane) * GBKB + c * 16) =
                                    make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                // generic-proxy stores must be visible to the tensor core's (async proxy) reads
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
            it += o.nkb;
        }
    } else if (warp < GEPI_WARP0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(GREGS_MMA));
        if (warp == GMMA_WARP && lane == 0) {
            // ---------------- MMA issuer ----------------
            int it = 0, ch = 0;
            bool ok = true;
            int nkb = 0, bn = 64, nnkb = 0, nbn = 64;
            if (int(blockIdx.x) < ntiles) { nnkb = tiles[blockIdx.x].nkb; nbn = tiles[blockIdx.x].bn; }
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                nkb = nnkb;
                bn = nbn;
                if (t + int(gridDim.x) < ntiles) { nnkb = tiles[t + gridDim.x].nkb; nbn = tiles[t + gridDim.x].bn; }
                const uint32_t idesc = instr_desc(false, BM, bn);
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int kin = kb % GCHUNK, buf = ch & 1;
                    if (kin == 0 && ch >= 2) {  // the epilogue has drained this buffer's previous chunk
                        if (!mbar_wait(&tempty[buf], ((ch >> 1) - 1) & 1, err, 32)) { ok = false; break; }
                        tc_fence_after();
                    }
                    const int s = it % C::STAGES;
                    if (!mbar_wait(&full[s], (it / C::STAGES) & 1, err, 33)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * C::STAGE_BYTES);
                    const uint32_t sb = sa + TERMS * C::A_PLANE;
#pragma unroll
                    for (int ks = 0; ks < GBKB / 32; ++ks) {
#pragma unroll
                        for (int pi = 0; pi < C::NPROD; ++pi) {
                            int p, q, collector;
                            product<TERMS, false>(pi, p, q, collector);
                            const uint32_t accumulate = (kin > 0 || ks > 0 || pi > 0) ? 1u : 0u;
                            const uint64_t ad = smem_desc(sa + p * C::A_PLANE + ks * 32, 8 * GBKB, 4);
                            const uint64_t bd = smem_desc(sb + q * C::B_PLANE + ks * 32, 8 * GBKB, 4);
                            umma<false>(tmem + uint32_t(buf * GBN), ad, bd, idesc, accumulate, collector);
                        }
                    }
                    umma_commit(&empty[s]);
                    *slabs_done = it + 1;
                    if (kin == GCHUNK - 1 || kb == nkb - 1) {
                        umma_commit(&tfull[buf]);
                        ++ch;
                    }
                }
            }
            *slabs_done = 0x7fffffff;  // also after an expired wait
        } else if (warp > GMMA_WARP) {
            // ---------------- prefetch: every third slab each ----------------
            int first = 0, done = 0, mine = warp - GMMA_WARP - 1;  // slabs before the tile; this warp's next one
            for (int t = blockIdx.x; t < ntiles && done < 0x7fffffff; t += gridDim.x) {
                const int nkb = tiles[t].nkb;
                for (; mine < first + nkb; mine += GPREFETCH_WARPS) {
                    for (int tries = 0; done < mine - C::AHEAD && tries < 100000; ++tries) {
                        done = *slabs_done;
                        if (done < mine - C::AHEAD) __nanosleep(50);
                    }
                    if (done < mine - C::AHEAD) done = 0x7fffffff;  // no progress: only the prefetches end
                    if (done == 0x7fffffff) break;
                    if (mine >= done + GGROUPS) prefetch_slab(tiles + t, mine - first, nkb, lane);
                }
                first += nkb;
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(GREGS_EPI));
        const int quarter = warp & 3;  // the TMEM lanes this warp may read
        const int part = (warp - GEPI_WARP0) >> 2;
        int ch = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const TcTile* d = tiles + t;
            const int nkb = d->nkb, epi_cols = d->bn / 2, rows = d->rows, cols = d->cols;
            const i64 ldc = d->ldc;
            float* const corner = d->c;
            const float alpha = d->alpha, beta = d->beta;
            const int row = quarter * 32 + lane, c0 = part * epi_cols;
            float acc[GBN / 2];
#pragma unroll
            for (int j = 0; j < GBN / 2; ++j) acc[j] = 0.0f;
            const int nchunks = (nkb + GCHUNK - 1) / GCHUNK;
            for (int c = 0; c < nchunks && ok; ++c, ++ch) {
                const int buf = ch & 1;
                if (!mbar_wait(&tfull[buf], (ch >> 1) & 1, err, 34)) { ok = false; break; }
                tc_fence_after();
                const uint32_t base = tmem + (uint32_t(quarter * 32) << 16) + uint32_t(buf * GBN + c0);
#pragma unroll
                for (int e = 0; e < GBN / 2; e += 16) {
                    if (e < epi_cols) {  // warp-uniform
                        uint32_t rr[16];
                        tmem_ld16(base + uint32_t(e), rr);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[e + j] += __uint_as_float(rr[j]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tempty[buf]);
            }
            if (!ok) break;
            const int nc = row < rows ? min(epi_cols, cols - c0) : 0;  // live columns of this thread (may be negative)
            float* cp = corner + row + i64(c0) * ldc;
            if (beta == 0.0f) {
#pragma unroll
                for (int j = 0; j < GBN / 2; ++j, cp += ldc) st_if(cp, alpha * acc[j], j < nc);
            } else {
                // eight loads of C before their stores (a store may alias any later load)
#pragma unroll
                for (int j0 = 0; j0 < GBN / 2; j0 += 8) {
                    float cv[8];
                    const float* q = cp;
#pragma unroll
                    for (int j = 0; j < 8; ++j, q += ldc) cv[j] = j0 + j < nc ? *q : 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j, cp += ldc)
                        st_if(cp, fmaf(beta, cv[j], alpha * acc[j0 + j]), j0 + j < nc);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == GMMA_WARP) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem, 2 * GBN);
    }
}

}  // namespace gtc

// ---- plans (called by grouped.cu) -------------------------------------------------
// The device table holds TcTile[ntiles].

// Builds the device table of a grouped split sgemm: per problem its tile width (from
// the tuning table's size class), its tiles ordered by reduction length, longest first.
int grouped_tc_build(int terms, int count, const mbg_sgemm_problem* probs, GroupedTcPlan& out) {
    using namespace gtc;
    struct Place {  // what is sorted: the descriptors are five times as large
        int prob, tm, tn, nkb;
    };
    std::vector<Place> order;
    order.reserve(size_t(count) * 4);
    out.terms = terms;
    out.count = 0;
    for (int i = 0; i < count; ++i) {
        const mbg_sgemm_problem& q = probs[i];
        if (q.m == 0 || q.n == 0) continue;
        ++out.count;
        const i64 nkb = k_slabs(q.alpha == 0.0f ? 0 : q.k, GBK).n;
        const i64 tn = cdiv(q.n, grouped_tc_tile_cols(q.m, q.n, q.k, is_t(q.trans_a), is_t(q.trans_b))), tm = cdiv(q.m, BM);
        // (k > 2^36: one row of op(A) takes 256 GB)
        if (nkb > 0x7fffffff || tm > 0x3fffffff || tn > 0x3fffffff || tm * tn > 0x3fffffff) return MBG_ERR_UNSUPPORTED;
        for (int n = 0; n < int(tn); ++n)
            for (int m = 0; m < int(tm); ++m) order.push_back(Place{i, m, n, int(nkb)});
    }
    if (order.size() > 0x3fffffff) return MBG_ERR_UNSUPPORTED;
    std::stable_sort(order.begin(), order.end(), [](const Place& x, const Place& y) { return x.nkb > y.nkb; });
    out.ntiles = int(order.size());
    if (out.ntiles == 0) return MBG_OK;
    std::vector<TcTile> t(order.size());
    for (size_t i = 0; i < order.size(); ++i) {
        const mbg_sgemm_problem& q = probs[order[i].prob];
        const bool ta = is_t(q.trans_a), tb = is_t(q.trans_b);
        TcTile& d = t[i];
        d.bn = grouped_tc_tile_cols(q.m, q.n, q.k, ta, tb);
        const i64 m0 = i64(order[i].tm) * BM, n0 = i64(order[i].tn) * d.bn;
        d.nkb = order[i].nkb;
        d.last = k_slabs(d.nkb ? q.k : 0, GBK).last;
        d.lda = q.lda; d.ldb = q.ldb; d.ldc = q.ldc;
        d.a = q.a + (d.nkb ? (ta ? m0 * q.lda : m0) : 0);
        d.b = q.b + (d.nkb ? (tb ? n0 : n0 * q.ldb) : 0);
        d.c = q.c + m0 + n0 * q.ldc;
        d.kcontig = (ta ? 1 : 0) | (tb ? 0 : 2);
        if (ta && q.lda % 2 == 0 && reinterpret_cast<uintptr_t>(d.a) % 8 == 0) d.kcontig |= 4;
        if (!tb && q.ldb % 2 == 0 && reinterpret_cast<uintptr_t>(d.b) % 8 == 0) d.kcontig |= 8;
        d.rows = int(imin(i64(BM), q.m - m0));
        d.cols = int(imin(i64(d.bn), q.n - n0));
        d.alpha = q.alpha; d.beta = q.beta;
    }
    const size_t bytes = sizeof(TcTile) * t.size();
    MBG_CUDA(cudaMalloc(&out.table, bytes));
    MBG_CUDA(cudaMemcpy(out.table, t.data(), bytes, cudaMemcpyHostToDevice));
    int dev = 0, sms = 148;
    MBG_CUDA(cudaGetDevice(&dev));
    MBG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    out.grid = int(imin(out.ntiles, sms));
    // the wait-error flag is created now: its first use must not fall inside the plan's graph capture
    out.err = device_error_flag();
    const int smem = terms == 3 ? GCfg<3>::SMEM_BYTES : GCfg<2>::SMEM_BYTES;
    if (terms == 3)
        MBG_CUDA(cudaFuncSetAttribute(grouped_tc_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    else
        MBG_CUDA(cudaFuncSetAttribute(grouped_tc_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return MBG_OK;
}

int grouped_tc_enqueue(const GroupedTcPlan& p, cudaStream_t s) {
    using namespace gtc;
    if (p.ntiles == 0) return MBG_OK;
    const TcTile* t = static_cast<const TcTile*>(p.table);
    if (p.terms == 3) grouped_tc_kernel<3><<<p.grid, GTHREADS, GCfg<3>::SMEM_BYTES, s>>>(t, p.ntiles, p.err);
    else grouped_tc_kernel<2><<<p.grid, GTHREADS, GCfg<2>::SMEM_BYTES, s>>>(t, p.ntiles, p.err);
    return check_launch("grouped_sgemm_tc");
}

void grouped_tc_free(GroupedTcPlan& p) {
    if (p.table) cudaFree(p.table);
    p.table = nullptr;
}

}  // namespace mbg
