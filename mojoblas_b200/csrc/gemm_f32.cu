// Plain FP32 GEMM on the CUDA cores, 128 x 128 or 64 x 64 tiles — the single-precision
// drop-in arithmetic for mojoBLAS gemm (src/level3/gemm.mojo:56-377, v11
// :2092-2436) and, with a triangular tile schedule, ssyrk
// (src/level3/syrk.mojo:20-200).
//
// One CTA per 128 x 128 tile of C; launches that would fill fewer than two waves of those
// may take 64 x 64 tiles and a cluster of CTAs per tile; the tile code (cp.async pipeline,
// register blocking, epilogue) is gemm_f32_tile.cuh, shared with the grouped
// sgemm plans.
#include "mbg_internal.cuh"
#include "gemm_f32_tile.cuh"

namespace mbg {

namespace {

using namespace f32t;

template <int FT, bool TA, bool TB, int TRI, bool VA, bool VB, class Slab>
__global__ void __launch_bounds__(FNT, FT == 128 ? 2 : 4)
gemm_f32_kernel(i64 m, i64 n, i64 k, float alpha, const float* __restrict__ A, i64 lda,
                const float* __restrict__ B, i64 ldb, float beta, float* __restrict__ C, i64 ldc, int band) {
    extern __shared__ __align__(16) float fsm[];
    pdl_wait();  // (and no pdl_next: launch_pdl)
    i64 tm, tn;
    if (TRI == 0) {
        tm = blockIdx.x;
        tn = blockIdx.y;
        band_order(band, tm, tn);
    } else {
        i64 ti, tj;
        f32_tri_tile(blockIdx.x, ti, tj);
        if (TRI == 1) { tm = ti; tn = tj; } else { tm = tj; tn = ti; }
    }
    f32_tile<FT, TA, TB, TRI, VA, VB, false, Slab>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, tm, tn, fsm, band);
}


// A cluster of CTAs per tile (f32_tile, CK): a product with few tiles spreads its reduction
// over the SMs they leave idle.
template <int FT, bool TA, bool TB, bool VA, bool VB>
__global__ void __launch_bounds__(FNT, FT == 128 ? 2 : 4)
gemm_f32_ck_kernel(i64 m, i64 n, i64 k, float alpha, const float* __restrict__ A, i64 lda,
                   const float* __restrict__ B, i64 ldb, float beta, float* __restrict__ C, i64 ldc, unsigned tiles_m,
                   int unit) {
    extern __shared__ __align__(16) float fsm[];
    pdl_wait();  // (and no pdl_next: launch_pdl)
    const unsigned tile = blockIdx.x / clu::size();
    f32_tile<FT, TA, TB, 0, VA, VB, true>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, tile % tiles_m, tile / tiles_m,
                                          fsm, KB_NONE, unit);
}

template <int FT, bool TA, bool TB, bool VA, bool VB>
int launch_f32_ck_t(int S, int unit, i64 m, i64 n, i64 k, float alpha, const float* a, i64 lda, const float* b, i64 ldb,
                    float beta, float* c, i64 ldc) {
    constexpr size_t SM = f32_ck_smem<FT>();
    static std::atomic<unsigned> configured{0};  // one bit per device
    int dev = 0;
    MBG_CUDA(cudaGetDevice(&dev));
    if (!configured_on(configured, dev)) {
        MBG_CUDA(cudaFuncSetAttribute(gemm_f32_ck_kernel<FT, TA, TB, VA, VB>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM));
        mark_configured(configured, dev);
    }
    const unsigned gm = unsigned(cdiv(m, FT));
    const clu::Launch l(gm * unsigned(cdiv(n, FT)) * unsigned(S), S, FNT, SM, stream(), true);
    MBG_CUDA(cudaLaunchKernelEx(&l.cfg, gemm_f32_ck_kernel<FT, TA, TB, VA, VB>, m, n, k, alpha, a, lda, b, ldb, beta,
                                c, ldc, gm, unit));
    return check_launch("gemm_f32");
}

template <int FT>
int launch_f32_ck(int S, int unit, bool ta, bool tb, i64 m, i64 n, i64 k, float alpha, const float* a, i64 lda,
                  const float* b, i64 ldb, float beta, float* c, i64 ldc) {
    const bool va = f32_vec(!ta, a, lda), vb = f32_vec(tb, b, ldb);
#define CKL(TA_, TB_, VA_, VB_) \
    return launch_f32_ck_t<FT, TA_, TB_, VA_, VB_>(S, unit, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc)
    if (!ta && tb) {
        if (va && vb) CKL(false, true, true, true);
        if (va) CKL(false, true, true, false);
        if (vb) CKL(false, true, false, true);
        CKL(false, true, false, false);
    }
    if (!ta) {
        if (va) CKL(false, false, true, false);
        CKL(false, false, false, false);
    }
    if (tb) {
        if (vb) CKL(true, true, false, true);
        CKL(true, true, false, false);
    }
    CKL(true, false, false, false);
#undef CKL
}

// Tile and CTAs per tile of a product under two waves of 128-tiles, by the estimated time in
// microseconds.  A slab takes the longer of a CTA's own latency and its share of the SM: 0.51 and
// 0.46 for 64-tiles (16 deep), 2.75 for 128-tiles (32 deep), and 0.74, 0.64 and 3.15 where neither
// operand takes 16-byte copies; sharing a tile adds 1 + 0.2 S, and has to be worth a tenth.
// (Measured around each call, launch included: 512^3 NT 26.9 us on 64-tiles, 17.7 with four CTAs
// each; 64 x 64 x 1000 TT 54.9 and, with eight, 14.7; 1000^3 NN 91 on 64-tiles, 68 on 128-tiles
// with two.)
struct F32Shape {
    int ft, S;
    int unit;  // slabs that a CTA's part of the reduction is a multiple of
};
inline F32Shape f32_shape(i64 m, i64 n, i64 k, int vec_operands, int S_min, int S_max) {
    F32Shape best{64, S_min, 1};
    double t_best = 0;
    const double scalar = (2 - vec_operands) / 2.0;
    for (int ft = 64; ft <= 128; ft *= 2) {
        const i64 tiles = cdiv(m, ft) * cdiv(n, ft), slabs = cdiv(k, ft == 128 ? Deep<128>::K : Deep<64>::K);
        const double lat = ft == 128 ? 2.75 + 0.4 * scalar : 0.51 + 0.23 * scalar;
        const double rate = ft == 128 ? lat : 0.46 + 0.18 * scalar;
        for (int S = S_min; S <= S_max && S <= slabs; ++S) {
            const double share = rate * double(cdiv(tiles * S, clu::usable_sms(S)));
            double t = double(cdiv(slabs, S)) * (share > lat ? share : lat) + (S > 1 ? 1.0 + 0.2 * S : 0.0);
            if (ft == 128 || S > 1) t *= 1.1;
            if (t_best == 0 || t < t_best) {
                t_best = t;
                best = F32Shape{ft, S, 1};
            }
        }
    }
    return best;
}

// The shape of a call.  At sizes that the pipelined host path takes, its column blocks and the call over all
// of C (on device pointers) have to divide a reduction alike, so the parts go by the whole
// product and by no alignment (staged copies have leading dimensions of their own).  The tile changes
// no sum and goes by what runs here: 1024 x 4100 x 4096 on pinned host memory takes 2.33 ms so, and
// 3.32 with the whole product's 128-tiles, 48 of them in a block.
//
// A banded product (trmm) takes 64-tiles when it has few: its tiles' reductions differ in length, and smaller
// ones fill the chip more evenly (strmm L 2048 x 1024 198 us, 232 on the 128-tiles of f32_shape).
inline F32Shape f32_schedule(i64 m, i64 n, i64 k, int vec_operands, bool banded) {
    const i64 ns = schedule_columns(n);
    const bool host_sized = double(m) * double(ns) * double(k) >= double(1ll << 34);
    auto few = [&](i64 columns) { return cdiv(m, 128) * cdiv(columns, 128) < 2 * 148; };
    if (banded) return F32Shape{few(n) ? 64 : 128, 1, 1};
    F32Shape sh = few(ns) ? f32_shape(m, ns, k, host_sized ? 2 : vec_operands, 1, clu::MAX_CTAS)
                          : F32Shape{128, 1, 1};
    if (host_sized && few(n) && (sh.S == 1 || sh.ft == 128)) {
        const int ft = f32_shape(m, n, k, vec_operands, sh.S, sh.S).ft;
        sh = F32Shape{ft, sh.S, sh.S > 1 && ft == 64 ? Deep<128>::K / Deep<64>::K : 1};
    }
    return sh;
}

template <int FT, int TRI, bool VA, bool VB, class Slab>
int launch_f32_slab(bool ta, bool tb, dim3 grid, i64 m, i64 n, i64 k, float alpha, const float* a, i64 lda,
                    const float* b, i64 ldb, float beta, float* c, i64 ldc, int band) {
    constexpr size_t SM = f32_smem<FT, Slab>();
    static std::atomic<unsigned> configured{0};  // one bit per device: more than 48 KB of shared memory needs an opt-in
    int dev = 0;
    MBG_CUDA(cudaGetDevice(&dev));
    if (!configured_on(configured, dev)) {
        MBG_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<FT, false, false, TRI, VA, VB, Slab>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM));
        MBG_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<FT, false, true, TRI, VA, VB, Slab>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM));
        MBG_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<FT, true, false, TRI, VA, VB, Slab>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM));
        MBG_CUDA(cudaFuncSetAttribute(gemm_f32_kernel<FT, true, true, TRI, VA, VB, Slab>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM));
        mark_configured(configured, dev);
    }
    cudaStream_t s = stream();
#define F32(TA_, TB_)                                                                                                   \
    MBG_CUDA(launch_pdl(gemm_f32_kernel<FT, TA_, TB_, TRI, VA, VB, Slab>, grid, dim3(FNT), SM, s, m, n, k, alpha, a, lda, b, \
                        ldb, beta, c, ldc, band))
    if (!ta && !tb) F32(false, false);
    else if (!ta && tb) F32(false, true);
    else if (ta && !tb) F32(true, false);
    else F32(true, true);
#undef F32
    return check_launch("gemm_f32");
}

// 128-tiles take deep slabs where an operand takes 16-byte copies (element by element, the 32 copies of
// a slab per thread and operand spill: 4096^3 NT with odd leading dimensions 3.12 ms in slabs of 16, 3.73 in
// slabs of 32) and where the padding of k costs less than they save, a tenth with both operands so
// (4096 x 4096 x 40: 55 us, 62 as two slabs of 32; x 144 both 118) and a fiftieth with one (4096^3 NN with
// odd leading dimensions 3.02 and 2.98 ms; 4096 x 4096 x 144 139 and 149 us).
template <int FT, int TRI, bool VA, bool VB>
int launch_f32_v(bool ta, bool tb, dim3 grid, i64 m, i64 n, i64 k, float alpha, const float* a, i64 lda,
                 const float* b, i64 ldb, float beta, float* c, i64 ldc, int band) {
    if constexpr (FT == 128 && (VA || VB))
        if ((VA && VB ? 92 : 97) * cdiv(k, Deep<128>::K) * Deep<128>::K <= 100 * cdiv(k, Shallow::K) * Shallow::K)
            return launch_f32_slab<FT, TRI, VA, VB, Deep<128>>(ta, tb, grid, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
    return launch_f32_slab<FT, TRI, VA, VB, Shallow>(ta, tb, grid, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
}

template <int FT, int TRI>
int launch_f32(bool ta, bool tb, dim3 grid, i64 m, i64 n, i64 k, float alpha, const float* a, i64 lda,
               const float* b, i64 ldb, float beta, float* c, i64 ldc, int band = KB_NONE) {
    const bool va = f32_vec(!ta, a, lda), vb = f32_vec(tb, b, ldb);
    if (va && vb)
        return launch_f32_v<FT, TRI, true, true>(ta, tb, grid, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
    if (va)
        return launch_f32_v<FT, TRI, true, false>(ta, tb, grid, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
    if (vb)
        return launch_f32_v<FT, TRI, false, true>(ta, tb, grid, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
    return launch_f32_v<FT, TRI, false, false>(ta, tb, grid, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
}

// dst[j + i * ldd] = src[i + j * lds] for i < rows, j < cols (32 x 32 tiles through shared memory)
__global__ void f32_transpose_kernel(i64 rows, i64 cols, const float* __restrict__ src, i64 lds,
                                     float* __restrict__ dst, i64 ldd) {
    __shared__ float tile[32][33];
    const i64 i0 = (i64)blockIdx.x * 32, j0 = (i64)blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const i64 i = i0 + threadIdx.x, j = j0 + r;
        if (i < rows && j < cols) tile[r][threadIdx.x] = src[i + j * lds];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const i64 j = j0 + threadIdx.x, i = i0 + r;
        if (i < rows && j < cols) dst[j + i * ldd] = tile[threadIdx.x][r];
    }
}

int launch_f32_transpose(i64 rows, i64 cols, const float* src, i64 lds, float* dst, i64 ldd) {
    ProfScope prof("gemm_f32_transpose");
    dim3 g((unsigned)cdiv(rows, 32), (unsigned)cdiv(cols, 32)), blk(32, 8);
    if (g.y > 65535) return MBG_ERR_UNSUPPORTED;
    f32_transpose_kernel<<<g, blk, 0, stream()>>>(rows, cols, src, lds, dst, ldd);
    return check_launch("gemm_f32_transpose");
}

}  // namespace

// C := alpha op(A) op(B) + beta C (alpha != 0, k > 0): 128 x 128 tiles, or, when those would
// fill fewer than two waves, the tile and the CTAs per tile that f32_shape takes to be fastest.
// band (KB_*): one operand is a dense triangle; each tile runs its part of k.
// The tiles copy an operand 16 bytes at a time only when it is contiguous along m
// (op(A)) or n (op(B)), as in NT.  In a large call (m n k >= 2^30) an operand that is
// contiguous along k instead (A with 'T', B with 'N') is first transposed into a
// workspace (2 x 4 bytes per element against the GEMM's 2k flops per element of C);
// every element's sum is unchanged, the NT tiles run.
int sgemm_f32(char ta, char tb, i64 m, i64 n, i64 k, float alpha, const float* a, i64 lda, const float* b,
              i64 ldb, float beta, float* c, i64 ldc, int band) {
    if (double(m) * double(n) * double(k) >= double(1ll << 30) && (is_t(ta) || is_n(tb))) {
        Workspace wa, wb;
        if (is_t(ta)) {  // A is k x m (k contiguous): At = m x k
            const i64 ld = cdiv(m, 4) * 4;
            MBG_TRY(wa.reserve(sizeof(float) * size_t(ld) * size_t(k)));
            MBG_TRY(launch_f32_transpose(k, m, a, lda, wa.as<float>(), ld));
            a = wa.as<float>();
            lda = ld;
            ta = 'N';
        }
        if (is_n(tb)) {  // B is k x n (k contiguous): Bt = n x k, used as op(B) = Bt^T
            const i64 ld = cdiv(n, 4) * 4;
            MBG_TRY(wb.reserve(sizeof(float) * size_t(ld) * size_t(k)));
            MBG_TRY(launch_f32_transpose(k, n, b, ldb, wb.as<float>(), ld));
            b = wb.as<float>();
            ldb = ld;
            tb = 'T';
        }
        return sgemm_f32(ta, tb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, band);
    }
    ProfScope prof("gemm_f32");
    const i64 gm = cdiv(m, 128), gn = cdiv(n, 128);
    const F32Shape sh = f32_schedule(m, n, k, int(f32_vec(is_n(ta), a, lda)) + int(f32_vec(is_t(tb), b, ldb)), band != KB_NONE);
    if (sh.S > 1)
        return sh.ft == 128 ? launch_f32_ck<128>(sh.S, sh.unit, is_t(ta), is_t(tb), m, n, k, alpha, a, lda, b, ldb, beta, c, ldc)
                            : launch_f32_ck<64>(sh.S, sh.unit, is_t(ta), is_t(tb), m, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
    if (sh.ft == 64) {
        const i64 sm = cdiv(m, 64), sn = cdiv(n, 64);
        if (sn > 65535 || sm > 0x7fffffff) return MBG_ERR_UNSUPPORTED;
        return launch_f32<64, 0>(is_t(ta), is_t(tb), dim3((unsigned)sm, (unsigned)sn), m, n, k, alpha, a, lda, b,
                                 ldb, beta, c, ldc, band);
    }
    if (gn > 65535 || gm > 0x7fffffff) return MBG_ERR_UNSUPPORTED;
    return launch_f32<128, 0>(is_t(ta), is_t(tb), dim3((unsigned)gm, (unsigned)gn), m, n, k, alpha, a, lda, b,
                              ldb, beta, c, ldc, band);
}

// Lower ('L') or upper triangle of C := alpha op(A) op(B) + beta C (ssyrk).
int sgemmt_f32(char uplo, char ta, char tb, i64 n, i64 k, float alpha, const float* a, i64 lda,
               const float* b, i64 ldb, float beta, float* c, i64 ldc) {
    ProfScope prof("gemm_f32");
    const i64 t = cdiv(n, 128);
    const i64 tiles = t * (t + 1) / 2;
    if (tiles > 0x7fffffff) return MBG_ERR_UNSUPPORTED;
    if (is_l(uplo))
        return launch_f32<128, 1>(is_t(ta), is_t(tb), dim3((unsigned)tiles), n, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
    return launch_f32<128, 2>(is_t(ta), is_t(tb), dim3((unsigned)tiles), n, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
}

}  // namespace mbg
