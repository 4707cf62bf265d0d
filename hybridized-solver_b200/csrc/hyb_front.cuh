// hyb_front.cuh - pivot work of one elimination level: the LU of a diagonal block and the
// solve of one strip of its row's upper blocks, in one CTA (k_front).
//
// What bounds it: the chain of pivots. Step i of the LU cannot start before step i - 1 has
// produced its pivot, and an FP64 reciprocal (71 cycles), the quotient (24) and a fused
// multiply-add (8) in sequence make about 105 cycles per pivot however many threads take part
// (latencies measured with one warp on a B200); a step that first has to fetch its pivot row
// from another lane takes 200 to 350, in registers or through shared memory. So:
//  - the block is factored in panels of eight columns with a row per lane, four pivots at a time: the four pivot rows are read
//    by every lane, which factors them for itself, and there is no exchange inside the four;
//  - the strip of the upper block is carried along as further columns of the block, so its
//    forward substitution is done when the LU is; while the panel is factored the other warps
//    apply the panel before to all columns beyond it (rank-8 products on the FP64 tensor
//    pipe, which has the FP64 units' rate but reads its operands once per 8x8 tile);
//  - every CTA of a pivot factors the block again (m^3 / 3 multiply-adds against the m^2 n of
//    a strip's update): a second launch and the trip of the factors through memory would cost
//    more than the arithmetic.
// The factorization of FP32 factors (T = float) runs in FP64 as well and rounds once, when
// the results are stored: an FP32 reciprocal is no shorter (77 cycles), so FP32 would save no
// time on the chain and would need a second, FP64 path for pivots with growth.
// Measured on a B200 in one CTA, in SM cycles: a 64x64 block 17.5k for the LU with a strip's
// forward part and 10.7k for its backward part (16 columns; 21k and 14k with 64), where the
// 256-thread kernels took 69k for the FP64 LU alone and 38k for a strip of 64; 16x16 3.7k and
// 2.5k. Factorization time of whole meshes, before and after: 25x25 p=6 53.0 to 16.2 ms, 24x24
// p=8 44.5 to 21.3 ms, 32x32 of orders 2..10 123 to 55 ms, 16x16 p=4 5.6 to 2.8 ms. The factors
// of both are the same but for the rounding of 33- to 64-row pivots.
#pragma once

#include "hyb_kernels.cuh"

namespace hyb
{

constexpr int kFrontThreads = 256;
constexpr int kFrontMax = 128; // largest pivot
constexpr int kPanel = 8;
constexpr int kLdStrip = 68; // row stride of the strip: 4 mod 16 doubles, conflict-free DMMA operands

// The block and the strip are held with their rows rounded up to 16.
__host__ __device__ constexpr int front_rows(int m)
{
    return (m + 15) / 16 * 16;
}

// Dynamic shared memory for pivots of up to m rows: the block (row stride 4 mod 16 doubles), the strip,
// the pivots' reciprocals and eight pivot rows of a panel.
__host__ __device__ constexpr int front_smem(int m)
{
    return (front_rows(m) * (front_rows(m) + 4) + front_rows(m) * kLdStrip + front_rows(m) + kPanel * kPanel) * 8;
}

// 1 / p to within an ulp for a pivot that is not extreme: the hardware's approximation (PTX
// rcp.approx.ftz.f64) refined by the first terms of 1 / (1 - e) = 1 + e + e^2 + ..., e = 1 - p r its
// error. No branch, so that the compiler can schedule a panel's steps into one another: with
// the operator / and its test for special values a step took 196 cycles.
__device__ __forceinline__ double front_reciprocal(double p)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(p));
    const double e = fma(-p, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// a / p from r = front_reciprocal(p): the product corrected once by its residual (Markstein, IBM J. Res.
// Dev. 34 (1990) 111), which is the correctly rounded quotient unless a / p lies within 2^-50 ulp of the
// middle between two values. A quotient that overflows gives NaN here; the callers look for
// values that are not finite and then divide.
__device__ __forceinline__ double front_quotient(double a, double p, double r)
{
    const double q = a * r;
    return fma(fma(-p, q, a), r, q);
}

// Pivots whose reciprocal overflows or loses digits, zeros, infinities and NaN: divided by outright.
__device__ __forceinline__ bool front_extreme(double p)
{
    const unsigned e = ((unsigned)__double2hiint(p) >> 20) & 0x7ff;
    return e - 23u >= 2000u; // |p| < 2^-1000 or >= 2^977
}

// front_panel by plain divisions, in shared memory: for extreme pivots and values that are not finite.
__device__ __noinline__ void front_panel_divide(double *d, int ld, int r0, int rows, int w)
{
    const int lane = threadIdx.x & 31;
    for (int c = r0; c < r0 + w; ++c)
    {
        const double p = d[c * ld + c];
        for (int r = c + 1 + lane; r < rows; r += 32)
        {
            const double l = d[r * ld + c] / p;
            d[r * ld + c] = l;
            for (int e = c + 1; e < r0 + kPanel; ++e)
                d[r * ld + e] = fma(-l, d[c * ld + e], d[r * ld + e]);
        }
        __syncwarp();
    }
}

// Barrier 1 among the first n threads.
__device__ __forceinline__ void front_sync(int n)
{
    if (n > 32)
        asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
    else
        __syncwarp();
}

// The warps that hold a row of a panel (a row per lane) factor the eight columns from r0 on of the rows
// r0 .. rows - 1 of d (row stride ld) in place, w of them in use (beyond, the block is the
// identity's). Pivots four at a time: their rows go through ubuf to every lane, and every lane
// factors them. rpiv: the pivots' reciprocals. The results are stored only when all are finite
// and no pivot is extreme; otherwise *bad, zero before, becomes r0 + 1, the columns are factored
// again with divisions and *extreme is set.
__device__ __forceinline__ void front_panel(double *d, int ld, int r0, int rows, int w, double *rpiv, double *ubuf,
                                            int *bad, int *extreme)
{
    const int t0 = threadIdx.x, nt = (rows - r0 + 31) & ~31;
    const bool mine = r0 + t0 < rows;
    double x[kPanel], rp[kPanel];
    double *own = d + (r0 + t0) * ld + r0;
#pragma unroll
    for (int c = 0; c < kPanel; c += 2)
    {
        const double2 v = mine ? *reinterpret_cast<const double2 *>(own + c) : make_double2(0, 0);
        x[c] = v.x;
        x[c + 1] = v.y;
    }
    bool no = false;
#pragma unroll
    for (int h = 0; h < kPanel; h += 4)
    {
        const double *ub = d + (r0 + h) * ld + r0; // the first four rows are as they were
        int ldu = ld;
        if (h > 0)
        {
            if (t0 >= h && t0 < h + 4)
#pragma unroll
                for (int e = h; e < kPanel; e += 2)
                    *reinterpret_cast<double2 *>(ubuf + t0 * kPanel + e) = make_double2(x[e], x[e + 1]);
            front_sync(nt);
            ub = ubuf + h * kPanel;
            ldu = kPanel;
        }
        double u[4][kPanel];
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = h; e < kPanel; e += 2)
            {
                const double2 v = *reinterpret_cast<const double2 *>(ub + t * ldu + e);
                u[t][e] = v.x;
                u[t][e + 1] = v.y;
            }
#pragma unroll
        for (int t = 0; t < 4; ++t)
        {
            const int c = h + t;
            const double p = u[t][c], r = front_reciprocal(p);
            no |= front_extreme(p);
            rp[c] = r;
#pragma unroll
            for (int i = t + 1; i < 4; ++i)
            {
                const double l = front_quotient(u[i][c], p, r);
#pragma unroll
                for (int e = c + 1; e < kPanel; ++e)
                    u[i][e] = fma(-l, u[t][e], u[i][e]);
            }
            // rows at or above the pivot keep their values
            const double l = front_quotient(x[c], p, r), f = t0 > c ? l : 0.0;
            x[c] = t0 > c ? l : x[c];
#pragma unroll
            for (int e = c + 1; e < kPanel; ++e)
                x[e] = fma(-f, u[t][e], x[e]);
        }
    }
    double sum = 0;
#pragma unroll
    for (int c = 0; c < kPanel; ++c)
        sum += x[c];
    if (no || !isfinite(sum))
        *bad = r0 + 1;
    front_sync(nt); // also: every warp has read the columns
    if (*reinterpret_cast<volatile int *>(bad) == r0 + 1)
    {
        if (t0 < 32)
            front_panel_divide(d, ld, r0, rows, w);
        if (t0 == 0)
            *extreme = 1;
        return;
    }
    if (mine)
#pragma unroll
        for (int c = 0; c < kPanel; c += 2)
            *reinterpret_cast<double2 *>(own + c) = make_double2(x[c], x[c + 1]);
    if (t0 == 0)
#pragma unroll
        for (int c = 0; c < kPanel; c += 2)
            *reinterpret_cast<double2 *>(rpiv + r0 + c) = make_double2(rp[c], rp[c + 1]);
}

// c -= a b on 8x8 tiles in shared memory with a contraction of eight, by one warp: the rows row0,
// row0 + 8, ... < rows of the column tile at c (row stride ldc), a (row stride lda) the eight
// columns of the same rows, b (row stride ldb) the eight rows of the column tile, the first kw of
// which count (what lies beyond the block's edge may be anything).
// kBatch tiles are loaded before the first is stored: their latencies overlap. With kDown the
// contraction runs from the last of the eight down, the order of a backward substitution.
template <int kBatch, bool kDown = false>
__device__ __forceinline__ void front_tiles(double *c, int ldc, const double *a, int lda, const double *b, int ldb,
                                            int row0, int rows, int kw = kPanel)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int k0 = kDown ? 7 - q : q, k1 = kDown ? 3 - q : 4 + q;
    const double b0 = k0 < kw ? b[k0 * ldb + g] : 0.0, b1 = k1 < kw ? b[k1 * ldb + g] : 0.0;
    double *pc = c + (row0 + g) * ldc + 2 * q;
    const double *pa = a + (row0 + g) * lda;
#pragma unroll 1
    for (int r = row0; r < rows; r += 8 * kBatch, pc += 8 * kBatch * ldc, pa += 8 * kBatch * lda)
    {
        double2 v[kBatch];
        double a0[kBatch], a1[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
            if (i == 0 || r + 8 * i < rows)
            {
                v[i] = *reinterpret_cast<double2 *>(pc + 8 * i * ldc);
                a0[i] = pa[8 * i * lda + k0];
                a1[i] = pa[8 * i * lda + k1];
            }
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
            if (i == 0 || r + 8 * i < rows)
            {
                dmma_8x8x4(v[i].x, v[i].y, k0 < kw ? -a0[i] : 0.0, b0);
                dmma_8x8x4(v[i].x, v[i].y, k1 < kw ? -a1[i] : 0.0, b1);
            }
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
            if (i == 0 || r + 8 * i < rows)
                *reinterpret_cast<double2 *>(pc + 8 * i * ldc) = v[i];
    }
}

// Eight rows of one column (stride ld) <- L^{-1} of them, L the unit lower block at d (row stride ldd).
// Rows and columns beyond the block's edge only reach rows beyond it.
__device__ __forceinline__ void front_forward(const double *d, int ldd, double *col, int ld)
{
    double x[kPanel];
#pragma unroll
    for (int i = 0; i < kPanel; ++i)
        x[i] = col[i * ld];
#pragma unroll
    for (int k = 0; k < kPanel - 1; ++k)
#pragma unroll
        for (int i = k + 1; i < kPanel; ++i)
            x[i] = fma(-d[i * ldd + k], x[k], x[i]);
#pragma unroll
    for (int i = 1; i < kPanel; ++i)
        col[i * ld] = x[i];
}

// The same with the upper block, its pivots' reciprocals and the first w rows. Returns whether the
// results are finite; they are stored only then (kDivide: always).
template <bool kDivide>
__device__ __forceinline__ bool front_backward(const double *d, int ldd, const double *rpiv, double *col, int ld, int w)
{
    double x[kPanel], sum = 0;
#pragma unroll
    for (int i = 0; i < kPanel; ++i)
        x[i] = i < w ? col[i * ld] : 0.0;
#pragma unroll
    for (int k = kPanel - 1; k >= 0; --k)
    {
        if (k >= w) // uniform
            continue;
        const double p = d[k * ldd + k];
        x[k] = kDivide ? x[k] / p : front_quotient(x[k], p, rpiv[k]);
        sum += x[k];
#pragma unroll
        for (int i = 0; i < k; ++i)
            x[i] = fma(-d[i * ldd + k], x[k], x[i]);
    }
    if (!kDivide && !isfinite(sum))
        return false;
#pragma unroll
    for (int i = 0; i < kPanel; ++i)
        col[i * ld] = x[i];
    return true;
}

__device__ __noinline__ void front_backward_divide(const double *d, int ldd, double *col, int ld, int w)
{
    front_backward<true>(d, ldd, nullptr, col, ld, w);
}

// Loads rows x cols values of a row-major block (row stride lds) into shared memory (row stride ld),
// as doubles, zero up to prows x pcols (pcols at most 64); warp `warp` of nw. Sixteen values per
// lane are in flight at once. Returns the largest magnitude.
template <typename T>
__device__ __forceinline__ double front_load(double *dst, int ld, const T *src, int lds, int rows, int cols, int prows,
                                             int pcols, int warp, int nw)
{
    const int lane = threadIdx.x & 31;
    double amax = 0;
    for (int r0 = warp; r0 < prows; r0 += 8 * nw)
    {
        double v[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int r = r0 + i * nw, c = lane + 32 * h;
                v[i][h] = r < rows && c < cols ? (double)src[(int64_t)r * lds + c] : 0.0;
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int r = r0 + i * nw, c = lane + 32 * h;
                if (r < prows && c < pcols)
                    dst[r * ld + c] = v[i][h];
                amax = fmax(amax, fabs(v[i][h]));
            }
    }
    return amax;
}

// LU of the m x m block d in shared memory (row stride ldd, continued by the identity up to the
// next multiple of 16) and, as further columns, b <- L^{-1} b for the nb tiles of eight columns of
// the strip b. `load_strip` (called by the warps other than the first, with their number among
// them and their count) fills b before it is first read; it runs beside the first panel.
template <typename F>
__device__ __forceinline__ void front_factor(double *d, int ldd, int m, double *b, int nb, double *rpiv, double *ubuf,
                                             int *flags, F load_strip)
{
    const int tid = threadIdx.x, warp = tid >> 5, nw = kFrontThreads / 32;
    const int rows = (m + kPanel - 1) / kPanel * kPanel;
    for (int r0 = 0; r0 < rows; r0 += kPanel)
    {
        const int r1 = r0 + kPanel, w = min(kPanel, m - r0);
        const int np = (rows - r0 + 31) / 32; // warps on the panel
        if (warp < np)
        {
            front_panel(d, ldd, r0, rows, w, rpiv, ubuf, flags, flags + 1);
        }
        else if (r0 == 0)
        {
            load_strip(warp - np, nw - np);
        }
        else
        {
            // the panel before on the columns beyond this one, in units of a column tile and up to four rows of tiles
            const int nd = (rows - r1) / 8, k0 = r0 - kPanel, nc = nd + nb;
            for (int t = warp - np; t < nc * ((rows - r0 + 31) / 32); t += nw - np)
            {
                const int i = t % nc, row = r0 + t / nc * 32;
                double *c = i < nd ? d + r1 + 8 * i : b + 8 * (i - nd);
                const int ldc = i < nd ? ldd : kLdStrip;
                front_tiles<4>(c, ldc, d + k0, ldd, c + k0 * ldc, ldc, row, min(row + 32, rows));
            }
        }
        __syncthreads();
        // the panel's rows in every column beyond it
        const int nd = rows - r1;
        for (int t = tid; t < nd + 8 * nb; t += kFrontThreads)
        {
            const int ldc = t < nd ? ldd : kLdStrip;
            front_forward(d + r0 * ldd + r0, ldd, t < nd ? d + r0 * ldd + r1 + t : b + r0 * kLdStrip + t - nd, ldc);
        }
        __syncthreads();
        // the next panel's columns, so that it can start
        if (nd > 0)
        {
            for (int row = r1 + 8 * warp; row < rows; row += 8 * nw)
                front_tiles<1>(d + r1, ldd, d + r0, ldd, d + r0 * ldd + r1, ldd, row, row + 8);
            __syncthreads();
        }
    }
}

// b <- U^{-1} b for the strip, U the upper factor in d. Two warps solve eight rows of the strip's
// columns while the others apply the eight rows below to the rows above them.
__device__ __forceinline__ void front_back(const double *d, int ldd, int m, double *b, int nb, const double *rpiv,
                                           bool extreme)
{
    const int tid = threadIdx.x, warp = tid >> 5, nw = kFrontThreads / 32;
    for (int r0 = (m - 1) / kPanel * kPanel; r0 >= 0; r0 -= kPanel)
    {
        const int w = min(kPanel, m - r0), r1 = r0 + kPanel;
        if (warp < 2)
        {
            double *col = b + r0 * kLdStrip + tid;
            if (tid < 8 * nb && (extreme || !front_backward<false>(d + r0 * ldd + r0, ldd, rpiv + r0, col, kLdStrip, w)))
                front_backward_divide(d + r0 * ldd + r0, ldd, col, kLdStrip, w);
        }
        else if (r1 < m)
        {
            for (int t = warp - 2; t < nb * ((r0 + 31) / 32); t += nw - 2)
            {
                const int c0 = 8 * (t % nb), row = t / nb * 32;
                front_tiles<4, true>(b + c0, kLdStrip, d + r1, ldd, b + r1 * kLdStrip + c0, kLdStrip, row,
                                     min(row + 32, r0), min(kPanel, m - r1));
            }
        }
        __syncthreads();
        if (r0 == 0)
            break;
        for (int t = warp; t < nb; t += nw)
            front_tiles<1, true>(b + 8 * t, kLdStrip, d + r0, ldd, b + r0 * kLdStrip + 8 * t, kLdStrip, r0 - 8, r0, w);
        __syncthreads();
    }
}

// The level's pivots p0 .. p1 of up to 128 rows: grid.x the units of lu_pref (one per upper block
// of a pivot, at least one per pivot), grid.y the strips (of 16, 32 or 64 columns) of the widest upper block. Each
// CTA reads and factors its pivot's block; the one that takes the pivot's last ticket -- after
// all have read it -- writes the factors back. The first CTA of a pivot reports zero and
// non-finite pivots and, with a growth limit (the mixed form), whether the pivot's growth
// max|U| / max|D| passes it: counted as before by size, though the arithmetic is FP64 either way.
template <typename T>
__global__ void __launch_bounds__(kFrontThreads, 2)
    k_front(DevSym S, T *__restrict__ slab, int64_t p0, int64_t p1, int *__restrict__ tickets, int *status,
            float growth_limit, int strip)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_writer, s_flags[2]; // a panel to be divided by its pivots; any such
    const int tid = threadIdx.x;
    const int64_t u = S.lu_pref[p0] + blockIdx.x;
    const int64_t p = find_owner(S.lu_pref, p0, p1, u);
    const int64_t first = S.lu_pref[p], k = S.piv[p];
    const int64_t j = u - first, dpos = S.diag_pos[k], blk = dpos + 1 + j;
    const int m = S.size[k], rows = front_rows(m), ldd = rows + 4;
    const int cc = blk < S.row_ptr[k + 1] ? S.size[S.cols[blk]] : 0, col0 = strip * (int)blockIdx.y;
    const int w = max(0, min(strip, cc - col0)), nb = (w + 7) / 8;
    const int total = (int)(S.lu_pref[p + 1] - first) * (int)gridDim.y;
    const bool owner = j == 0 && blockIdx.y == 0;
    T *gd = slab + S.blk_off[dpos];
    T *gb = slab + S.blk_off[blk] + col0; // read only where w > 0 (blk_off has one entry more than blocks)
    double *d = reinterpret_cast<double *>(smem_raw);
    double *b = d + rows * ldd;
    double *rpiv = b + rows * kLdStrip, *ubuf = rpiv + rows;
    const int lane = tid & 31, warp = tid >> 5, nw = kFrontThreads / 32;

    double amax = 0;
    for (int c0 = 0; c0 < rows; c0 += 64)
        amax = fmax(amax, front_load(d + c0, ldd, gd + c0, m, m, m - c0, rows, min(64, rows - c0), warp, nw));
    for (int i = m + tid; i < rows; i += kFrontThreads)
        d[i * ldd + i] = 1;
    if (tid < 2)
        s_flags[tid] = 0;
    __syncthreads();
    if (tid == 0)
        s_writer = atomicAdd(tickets + p, 1) == total - 1;
    const bool check = owner && std::is_same_v<T, float> && growth_limit > 0;
    if (check)
        amax = cta_max(amax);
    if (w == 0 && !owner)
    {
        // a strip beyond this block's width: the factors may still be this CTA's to write
        __syncthreads();
        if (!s_writer)
            return;
    }
    front_factor(d, ldd, m, b, nb, rpiv, ubuf, s_flags,
                 [&](int wi, int n) { front_load(b, kLdStrip, gb, cc, m, w, rows, 8 * nb, wi, n); });
    if (nb > 0)
    {
        front_back(d, ldd, m, b, nb, rpiv, s_flags[1] != 0);
        for (int r = warp; r < m; r += nw)
            for (int c = lane; c < w; c += 32)
                gb[(int64_t)r * cc + c] = (T)b[r * kLdStrip + c];
    }
    if (s_writer)
    {
        for (int r = warp; r < m; r += nw)
            for (int c = lane; c < m; c += 32)
                gd[r * m + c] = (T)d[r * ldd + c];
        if (tid == 0)
            tickets[p] = 0; // ready for the next factorization
    }
    if (owner)
    {
        for (int i = tid; i < m; i += kFrontThreads)
        {
            const double v = d[i * ldd + i];
            if (v == 0 || !finite_val(v))
            {
                atomicAdd(status + (v == 0 ? ST_ZERO_PIVOTS : ST_NON_FINITE), 1);
                atomicMin(status + ST_FIRST_BAD, (int)k);
            }
        }
        if (check && lu_growth(d, m, ldd, amax) > (double)growth_limit && tid == 0)
            atomicAdd(status + (m <= 64 ? ST_GROWTH_FP64 : ST_GROWTH_KEPT), 1);
    }
}

} // namespace hyb
