// hyb_solve.cuh - substitution with the block factors (block_system_apply_operations and
// block_system_solve_u, src/blocks.c:729-800): forward y_k <- D_k^{-1} (y_k - sum_s L(k,s) y_s), then
// backward y_k <- y_k - sum_c U(k,c) y_c.
//
// What bounds it: the chain of pivots. y_k needs y_{k-1}, so every pivot costs at least one trip of
// a vector from one SM to another through L2, and whatever stands between the arrival of
// y_{k-1} and the departure of y_k. Both are kept short:
//  - a vector travels as tagged values -- value and tag of this solve and direction in one
//    store -- so a reader that sees the tag has the value: no fence, no flag, no second read;
//  - the nearest sources' blocks ("late": up to two) are handled apart from the others. Pivots of 16
//    to 128 rows keep W(k,s) = D_k^{-1} L(k,s) for them (k_late, after the factorization), so that
//    y_k = D_k^{-1} (y_k - sum of the others) - sum_late W(k,s) y_s: the substitution with D_k is
//    done while the late sources are still on their way, and only one product is left when
//    the last one arrives. W is solved for like U, with the same bound on the result's error as
//    substituting afterwards;
//  - the other ("early") blocks go in groups of up to eight to a CTA each, which adds their products in
//    registers as the sources arrive; the group nearest the pivot collects the others' sums.
// Measured on a B200, both directions, one right-hand side: see k_flow.
//
// Two forms with the same arithmetic (bit-identical results): k_flow, one cooperative launch per
// direction, and k_stage, one launch per level and direction.
#pragma once

#include "hyb_front.cuh"

namespace hyb
{

// A value with the tag of the solve direction that wrote it, stored and loaded whole.
template <typename T> struct Tagged;
template <> struct __align__(16) Tagged<double>
{
    double v;
    int64_t tag;
};
template <> struct __align__(8) Tagged<float>
{
    float v;
    int32_t tag;
};

__device__ __forceinline__ void tag_store(Tagged<double> *p, double v, int tag)
{
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((int64_t)tag)
                 : "memory");
}

__device__ __forceinline__ void tag_store(Tagged<float> *p, float v, int tag)
{
    const uint64_t w = (uint64_t)(uint32_t)__float_as_int(v) | (uint64_t)(uint32_t)tag << 32;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}

__device__ __forceinline__ bool tag_load(const Tagged<double> *p, int tag, double &v)
{
    int64_t a, b;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double(a);
    return b == tag;
}

__device__ __forceinline__ bool tag_load(const Tagged<float> *p, int tag, float &v)
{
    uint64_t w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    v = __int_as_float((int)(uint32_t)w);
    return (int)(w >> 32) == tag;
}

// Waits until *p carries the tag, at most wait_ns; false (and ST_TIMEOUT) when the time ran out here or
// elsewhere. Waits that are not on the chain leave pauses.
template <typename T>
__device__ __forceinline__ bool tag_wait(const Tagged<T> *p, int tag, T &v, bool pause, int *status, uint64_t wait_ns)
{
    if (tag_load(p, tag, v))
        return true;
    const uint64_t t0 = global_ns();
    for (;;)
    {
        for (int i = 0; i < 32; ++i)
        {
            if (pause)
                __nanosleep(40);
            if (tag_load(p, tag, v))
                return true;
        }
        if (schedule_aborted(status) || global_ns() - t0 > wait_ns)
        {
            atomicOr(status + ST_TIMEOUT, 1);
            return false;
        }
    }
}

constexpr int kNoTag = -1; // carried by nothing

// How the blocks left (forward) or right (backward) of pivot k's diagonal are shared out. Position i counts
// them from the farthest to the nearest; items: the groups of early positions, then the late ones.
struct FlowRow
{
    int64_t k, base; // pivot; filled index of the first block
    int64_t w;       // forward: offset of the row's W blocks, -1 where it has none
    int m, nb, ne, ng;
};

template <bool kFwd> __device__ __forceinline__ FlowRow flow_row(const DevSym &S, int64_t k)
{
    FlowRow f;
    const int64_t d = S.diag_pos[k];
    f.k = k;
    f.m = S.size[k];
    f.w = kFwd ? S.w_off[k] : -1;
    f.base = kFwd ? S.row_ptr[k] : d + 1;
    f.nb = (int)(kFwd ? d - f.base : S.row_ptr[k + 1] - f.base);
    f.ne = f.nb - min(f.nb, kFwd && f.w < 0 ? 1 : kFlowLate);
    f.ng = (f.ne + kFlowGroup - 1) / kFlowGroup;
    return f;
}

// Up to 16 columns of every row of one block in registers: thread t holds, of row r0 + t / tpr, the
// columns c0 + t % tpr + tpr c.
constexpr int kFlowRegs = 16;
template <typename T> struct FlowBlock
{
    T v[kFlowRegs];
    int64_t src; // unknowns before the source's
    int i, c0, K;
};

template <bool kFwd, typename T>
__device__ __forceinline__ void flow_load(FlowBlock<T> &g, const DevSym &S, const FlowRow &f, const T *__restrict__ slab,
                                          const T *__restrict__ wbuf, int i, int c0, int r0, int tpr)
{
    const int64_t blk = f.base + (kFwd ? i : f.nb - 1 - i);
    const int32_t s = S.cols[blk];
    g.i = i;
    g.c0 = c0;
    g.K = S.size[s];
    g.src = S.dof_off[s];
    const T *p = slab + S.blk_off[blk];
    if (kFwd && f.w >= 0 && i >= f.ne)
    {
        p = wbuf + f.w;
        for (int e = f.ne; e < i; ++e) // the late blocks before it
            p += (f.m * S.size[S.cols[f.base + e]] + kFlowPad - 1) / kFlowPad * kFlowPad;
    }
    const int row = r0 + (int)threadIdx.x / tpr, q = c0 + ((int)threadIdx.x & (tpr - 1));
    p += (int64_t)row * g.K + q;
    const bool in = row < f.m;
    if (c0 + kFlowRegs * tpr <= g.K)
    {
#pragma unroll
        for (int c = 0; c < kFlowRegs; ++c)
            g.v[c] = in ? p[c * tpr] : T(0);
    }
    else
    {
#pragma unroll
        for (int c = 0; c < kFlowRegs; ++c)
            g.v[c] = in && q + c * tpr < g.K ? p[c * tpr] : T(0);
    }
}

// Sums of a thread's products, NC right-hand sides at a time; with one, four sums side by side shorten the
// chain of additions.
template <typename T, int NC> struct FlowSum
{
    static constexpr int kWays = NC == 1 ? 4 : 1;
    T s[kWays][NC];
};

template <typename T, int NC>
__device__ __forceinline__ void flow_add(FlowSum<T, NC> &a, const FlowBlock<T> &g, const T *ybuf, int tpr)
{
    constexpr int W = FlowSum<T, NC>::kWays;
    const T *y = ybuf + (g.c0 + ((int)threadIdx.x & (tpr - 1))) * NC;
    const int left = g.K - g.c0 - ((int)threadIdx.x & (tpr - 1));
#pragma unroll
    for (int c = 0; c < kFlowRegs; ++c)
        if (c * tpr < left)
#pragma unroll
            for (int r = 0; r < NC; ++r)
                a.s[c % W][r] += g.v[c] * y[c * tpr * NC + r];
}

// The sums of a row's threads, in each of them.
template <typename T, int NC> __device__ __forceinline__ void flow_reduce(FlowSum<T, NC> &a, int tpr)
{
    constexpr int W = FlowSum<T, NC>::kWays;
#pragma unroll
    for (int r = 0; r < NC; ++r)
    {
        if constexpr (W == 4)
            a.s[0][r] = (a.s[0][r] + a.s[1][r]) + (a.s[2][r] + a.s[3][r]);
        for (int o = tpr >> 1; o > 0; o >>= 1)
            a.s[0][r] += __shfl_xor_sync(0xffffffffu, a.s[0][r], o);
    }
}

// Shared memory of a CTA of k_flow and k_stage, in values of T: two source vectors, a vector of the pivot's
// that is worked on, one that is kept, partial products of an inverse, and the diagonal block.
template <typename T> struct FlowSmem
{
    T *y[2], *acc, *z, *part, *d;
};

template <typename T> __device__ __forceinline__ FlowSmem<T> flow_smem(int max_m, int nc)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FlowSmem<T> s;
    T *p = reinterpret_cast<T *>(smem_raw);
    s.y[0] = p;
    s.y[1] = s.y[0] + max_m * nc;
    s.acc = s.y[1] + max_m * nc;
    s.z = s.acc + max_m * nc;
    s.part = s.z + max_m * nc;
    s.d = s.part + kThreads;
    return s;
}

template <typename T> __host__ __device__ constexpr int64_t flow_smem_bytes(int max_m, int nc, bool stage)
{
    return ((int64_t)4 * max_m * nc + kThreads + (stage ? (int64_t)max_m * (max_m | 1) : 0)) * (int64_t)sizeof(T);
}

// What a CTA prepares to apply D_k^{-1}: k's inverse in registers where the factorization left one (dinv
// set, 64 rows), else D_k in shared memory (stage) with an odd row stride.
template <typename T> struct FlowDiag
{
    static constexpr int kInv = std::is_same_v<T, float> ? kFlowRegs : 1; // only FP32 factors have inverses
    T inv[kInv];
    bool has_inv;
};

template <typename T>
__device__ __forceinline__ void flow_diag_load(FlowDiag<T> &g, const DevSym &S, const T *__restrict__ slab,
                                               const T *__restrict__ dinv, int64_t k, int m, T *sd, int stage)
{
    g.has_inv = std::is_same_v<T, float> && dinv && S.inv_idx[k] >= 0;
    if (g.has_inv)
    {
        const T *x = dinv + (int64_t)S.inv_idx[k] * 4096;
#pragma unroll
        for (int q = 0; q < FlowDiag<T>::kInv; ++q)
            g.inv[q] = x[q * kThreads + threadIdx.x];
    }
    else if (stage)
    {
        const T *gd = slab + S.blk_off[S.diag_pos[k]];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kThreads / 32;
#pragma unroll 4
        for (int r = warp; r < m; r += nw)
            for (int c = lane; c < m; c += 32)
                sd[r * (m | 1) + c] = gd[r * m + c];
    }
}

// acc <- D^{-1} acc for nc of NC columns by substitution (a function of its own: its registers are not
// needed while blocks are held).
template <typename T, int NC>
__device__ __noinline__ void flow_substitute(const T *d, int ldd, int m, T *acc, int nc)
{
    for (int r = threadIdx.x >> 5; r < nc; r += kThreads / 32)
    {
        if (m <= 32)
            warp_lu_solve<1>(d, ldd, m, acc, r, NC);
        else if (m <= 64)
            warp_lu_solve<2>(d, ldd, m, acc, r, NC);
        else if (m <= 96)
            warp_lu_solve1<3>(d, ldd, m, acc, r, NC);
        else if (m <= 128)
            warp_lu_solve1<4>(d, ldd, m, acc, r, NC);
        else
            warp_lu_solve_smem(d, ldd, m, acc, r, NC);
    }
}

// acc <- D_k^{-1} acc for nc of NC columns, by every thread of the CTA; acc is complete and in place after
// a barrier on both sides.
template <typename T, int NC>
__device__ __forceinline__ void flow_diag_solve(const FlowDiag<T> &g, const DevSym &S, const T *__restrict__ slab,
                                                int64_t k, int m, T *acc, T *part, const T *sd, int stage, int nc)
{
    const int tid = threadIdx.x;
    if constexpr (std::is_same_v<T, float>)
        if (g.has_inv)
        {
            // thread t holds X(t mod 64, 4 q + t / 64): four sums per row, added in a fixed order
            for (int c = 0; c < nc; ++c)
            {
                T s = T(0);
#pragma unroll
                for (int q = 0; q < kFlowRegs; ++q)
                    s += g.inv[q] * acc[(4 * q + (tid >> 6)) * NC + c];
                part[tid] = s;
                __syncthreads();
                if (tid < 64)
                    acc[tid * NC + c] = (part[tid] + part[64 + tid]) + (part[128 + tid] + part[192 + tid]);
                __syncthreads();
            }
            return;
        }
    flow_substitute<T, NC>(stage ? sd : slab + S.blk_off[S.diag_pos[k]], stage ? (m | 1) : m, m, acc, nc);
    __syncthreads();
}

// Dataflow substitution, one direction: a cooperative launch in which CTA b takes the items b, b + G, ...
// in order. Items are ordered by level (forward ascending, backward descending), a pivot's late item
// last; an item waits only for items before it and all CTAs are resident, so every wait ends; each
// is also bounded in time. ytag, ztag: dof x nrhs tagged values (the solution so far; a
// pivot's vector without its late sources, forward with D_k^{-1} applied where W exists); ptag:
// the sums of a pivot's early groups. The blocks of an item stream through two register
// buffers, the next one loaded while the present one waits for its source.
// withhold: pivot slot whose ztag is never written (fault injection), or -1.
template <typename T, int NC, bool kFwd>
__global__ void __launch_bounds__(kThreads, 2)
    k_flow(DevSym S, const T *__restrict__ slab, const T *__restrict__ wbuf, T *__restrict__ y, Tagged<T> *ytag,
           Tagged<T> *ztag, Tagged<T> *ptag, const T *__restrict__ dinv, int tag, int64_t n_items, int nrhs, int max_m,
           int stage, int64_t withhold, int *status, uint64_t wait_ns)
{
    const FlowSmem<T> sm = flow_smem<T>(max_m, NC);
    const int tid = threadIdx.x;
    for (int64_t j = blockIdx.x; j < n_items; j += gridDim.x)
    {
        const int64_t p = kFwd ? S.fwd_item_p[j] : S.bwd_item_p[j];
        const FlowRow f = flow_row<kFwd>(S, S.piv[p]);
        const int local = (int)(j - (kFwd ? S.fwdu_pref[p] : S.bwd_first[p])), m = f.m;
        const bool late = local == f.ng, last_group = local == f.ng - 1;
        const int i1 = late ? f.nb : f.ne - (f.ng - 1 - local) * kFlowGroup;
        const int i0 = late ? f.ne : max(0, i1 - kFlowGroup);
        const bool has_w = kFwd && f.w >= 0, held = p == withhold;
        // whether D_k^{-1} is applied here: before the late sources where W exists, else after them
        const bool solves = kFwd && (has_w ? last_group || (late && f.ng == 0) : late);
        const int64_t row_off = S.dof_off[f.k] * nrhs;
        Tagged<T> *part = ptag + (kFwd ? S.fwd_rows[p] : S.bwd_rows[p]) * nrhs;
        const int tpr = gemv_tpr<T>(m), rows = kThreads / tpr, q = tid & (tpr - 1);
        FlowDiag<T> dg;
        for (int ch = 0; ch < nrhs; ch += NC)
        {
            const int nc = min(NC, nrhs - ch);
            for (int r0 = 0; r0 < m; r0 += rows)
            {
                FlowBlock<T> g[2];
                if (i0 < i1)
                    flow_load<kFwd>(g[0], S, f, slab, wbuf, i0, 0, r0, tpr);
                if (solves && ch == 0 && r0 == 0)
                    flow_diag_load(dg, S, slab, dinv, f.k, m, sm.d, stage);
                __syncthreads(); // shared memory is free, D_k is staged
                bool ok = true;
                if (late && f.ng == 0 && r0 == 0)
                {
                    // no early blocks: the pivot's own values, solved at once where W exists
                    for (int e = tid; e < m * nc; e += kThreads)
                        sm.acc[e / nc * NC + e % nc] = y[row_off + (int64_t)(e / nc) * nrhs + ch + e % nc];
                    __syncthreads();
                    if (has_w)
                        flow_diag_solve<T, NC>(dg, S, slab, f.k, m, sm.acc, sm.part, sm.d, stage, nc);
                    for (int e = tid; e < m * NC; e += kThreads)
                        sm.z[e] = sm.acc[e];
                    if (held)
                    {
                        T v;
                        ok = tag_wait(ztag + row_off, kNoTag, v, true, status, wait_ns);
                    }
                }
                FlowSum<T, NC> a = {};
                int par = 0;
                // one step: prefetch the next piece, wait for this block's source, add
                auto step = [&](FlowBlock<T> &cur, FlowBlock<T> &nxt) {
                    int ni = cur.i, nc0 = cur.c0 + kFlowRegs * tpr;
                    if (nc0 >= cur.K)
                    {
                        ++ni;
                        nc0 = 0;
                    }
                    if (ni < i1)
                        flow_load<kFwd>(nxt, S, f, slab, wbuf, ni, nc0, r0, tpr);
                    if (cur.c0 == 0)
                    {
                        par ^= 1;
                        if (cur.i == i1 - 1 && (late ? f.ng > 0 : last_group && f.ng > 1))
                        {
                            // before the item's last source: what the pivot's other items have
                            for (int e = tid; e < m * nc && ok; e += kThreads)
                            {
                                const int64_t at = (int64_t)(e / nc) * nrhs + ch + e % nc;
                                T v, s = T(0);
                                if (late)
                                    ok = tag_wait(ztag + row_off + at, held ? kNoTag : tag, s, false, status, wait_ns);
                                else
                                    for (int h = 0; h < f.ng - 1 && ok; ++h)
                                    {
                                        ok = tag_wait(part + (int64_t)h * m * nrhs + at, tag, v, true, status, wait_ns);
                                        s = h == 0 ? v : s + v;
                                    }
                                sm.z[e / nc * NC + e % nc] = s;
                            }
                        }
                        const Tagged<T> *src = ytag + cur.src * nrhs + ch;
                        for (int e = tid; e < cur.K * nc && ok; e += kThreads)
                        {
                            T v;
                            ok = tag_wait(src + (int64_t)(e / nc) * nrhs + e % nc, tag, v, !late, status, wait_ns);
                            sm.y[par][e / nc * NC + e % nc] = v;
                        }
                        ok = __syncthreads_and(ok) != 0;
                    }
                    if (ok)
                        flow_add<T, NC>(a, cur, sm.y[par], tpr);
                    return ok && ni < i1;
                };
                if (i0 < i1)
                {
                    while (step(g[0], g[1]) && step(g[1], g[0]))
                        ;
                }
                else
                {
                    ok = __syncthreads_and(ok) != 0;
                }
                if (!ok)
                    return; // uniform
                flow_reduce<T, NC>(a, tpr);
                const int row = r0 + tid / tpr;
                if (q == 0 && row < m)
                {
#pragma unroll
                    for (int r = 0; r < NC; ++r)
                    {
                        if (r >= nc)
                            break;
                        const int64_t at = (int64_t)row * nrhs + ch + r;
                        const T s = a.s[0][r];
                        if (late)
                        {
                            const T v = i0 < i1 ? sm.z[row * NC + r] - s : sm.z[row * NC + r];
                            if (solves && !has_w)
                            {
                                sm.acc[row * NC + r] = v;
                            }
                            else
                            {
                                tag_store(ytag + row_off + at, v, tag);
                                y[row_off + at] = v;
                            }
                        }
                        else if (last_group)
                        {
                            const T v = y[row_off + at] - (f.ng > 1 ? sm.z[row * NC + r] + s : s);
                            if (solves)
                                sm.acc[row * NC + r] = v;
                            else
                                tag_store(ztag + row_off + at, v, tag);
                        }
                        else
                        {
                            tag_store(part + (int64_t)local * m * nrhs + at, s, tag);
                        }
                    }
                }
            }
            if (solves && !(late && has_w))
            {
                __syncthreads();
                flow_diag_solve<T, NC>(dg, S, slab, f.k, m, sm.acc, sm.part, sm.d, stage, nc);
                for (int e = tid; e < m * nc; e += kThreads)
                {
                    const int64_t at = (int64_t)(e / nc) * nrhs + ch + e % nc;
                    const T v = sm.acc[e / nc * NC + e % nc];
                    tag_store((late ? ytag : ztag) + row_off + at, v, tag);
                    if (late)
                        y[row_off + at] = v;
                }
            }
        }
    }
}

// The same, one level and direction per launch: CTA b takes item first + b of the level's items (all of whose
// sources are final), leaves its sums in `scratch` and takes a ticket of the pivot; the one that
// takes the last finishes the pivot with the arithmetic of k_flow.
template <typename T, int NC, bool kFwd>
__global__ void __launch_bounds__(kThreads, 2)
    k_stage(DevSym S, const T *__restrict__ slab, const T *__restrict__ wbuf, T *__restrict__ y, T *__restrict__ scratch,
            int *__restrict__ tickets, const T *__restrict__ dinv, int64_t first, int64_t rows0, int nrhs, int max_m,
            int stage)
{
    const FlowSmem<T> sm = flow_smem<T>(max_m, NC);
    const int tid = threadIdx.x;
    const int64_t j = first + blockIdx.x, p = kFwd ? S.fwd_item_p[j] : S.bwd_item_p[j];
    const FlowRow f = flow_row<kFwd>(S, S.piv[p]);
    const int local = (int)(j - (kFwd ? S.fwdu_pref[p] : S.bwd_first[p])), m = f.m, E = m * nrhs;
    const bool late = local == f.ng, has_w = kFwd && f.w >= 0;
    const int i1 = late ? f.nb : f.ne - (f.ng - 1 - local) * kFlowGroup;
    const int i0 = late ? f.ne : max(0, i1 - kFlowGroup);
    T *part = scratch + ((kFwd ? S.fwd_rows[p] : S.bwd_rows[p]) - rows0) * nrhs;
    T *yk = y + S.dof_off[f.k] * nrhs;
    const int tpr = gemv_tpr<T>(m), rows = kThreads / tpr, q = tid & (tpr - 1);
    for (int ch = 0; ch < nrhs; ch += NC)
    {
        const int nc = min(NC, nrhs - ch);
        for (int r0 = 0; r0 < m; r0 += rows)
        {
            FlowSum<T, NC> a = {};
            FlowBlock<T> g;
            for (int i = i0; i < i1; ++i)
            {
                __syncthreads();
                for (int c0 = 0; c0 == 0 || c0 < g.K; c0 += kFlowRegs * tpr)
                {
                    flow_load<kFwd>(g, S, f, slab, wbuf, i, c0, r0, tpr);
                    if (c0 == 0)
                    {
                        for (int e = tid; e < g.K * nc; e += kThreads)
                            sm.y[0][e / nc * NC + e % nc] = y[(g.src + e / nc) * nrhs + ch + e % nc];
                        __syncthreads();
                    }
                    flow_add<T, NC>(a, g, sm.y[0], tpr);
                }
            }
            flow_reduce<T, NC>(a, tpr);
            const int row = r0 + tid / tpr;
            if (q == 0 && row < m && f.nb > 0)
#pragma unroll
                for (int r = 0; r < NC; ++r)
                    if (r < nc)
                        part[(int64_t)local * E + (int64_t)row * nrhs + ch + r] = a.s[0][r];
        }
    }
    if (!last_ticket(tickets, p, f.ng + 1))
        return;
    FlowDiag<T> dg;
    if (kFwd)
        flow_diag_load(dg, S, slab, dinv, f.k, m, sm.d, stage);
    for (int ch = 0; ch < nrhs; ch += NC)
    {
        const int nc = min(NC, nrhs - ch);
        for (int e = tid; e < m * nc; e += kThreads)
        {
            const int64_t at = (int64_t)(e / nc) * nrhs + ch + e % nc;
            T v = yk[at];
            if (f.ng > 0)
            {
                T s = __ldcg(part + at);
                for (int h = 1; h < f.ng; ++h)
                    s += __ldcg(part + (int64_t)h * E + at);
                v -= s;
            }
            if (!has_w && f.nb > 0)
                v -= __ldcg(part + (int64_t)f.ng * E + at);
            sm.acc[e / nc * NC + e % nc] = v;
        }
        __syncthreads();
        if (kFwd)
            flow_diag_solve<T, NC>(dg, S, slab, f.k, m, sm.acc, sm.part, sm.d, stage, nc);
        for (int e = tid; e < m * nc; e += kThreads)
        {
            const int64_t at = (int64_t)(e / nc) * nrhs + ch + e % nc;
            T v = sm.acc[e / nc * NC + e % nc];
            if (has_w)
                v -= __ldcg(part + (int64_t)f.ng * E + at);
            yk[at] = v;
        }
        __syncthreads();
    }
}

// W(k,s) = D_k^{-1} L(k,s) for the late blocks of the pivots that keep them, in FP64, once the factors are
// final. grid.x: the W blocks, grid.y: their 64-column strips. Throughput only (one launch, off
// the chain): 0.1 ms per 1,000 blocks of 64x64 on a B200.
template <typename T>
__global__ void __launch_bounds__(kFrontThreads, 2) k_late(DevSym S, const T *__restrict__ slab, T *__restrict__ wbuf)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_extreme;
    const int64_t blk = S.w_blk[blockIdx.x];
    const int64_t k = S.w_row[blockIdx.x];
    const int m = S.size[k], K = S.size[S.cols[blk]], col0 = 64 * (int)blockIdx.y;
    if (col0 >= K)
        return;
    const int w = min(64, K - col0), nb = (w + 7) / 8, rows = front_rows(m), ldd = rows + 4;
    double *d = reinterpret_cast<double *>(smem_raw), *b = d + rows * ldd, *rpiv = b + rows * kLdStrip;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = kFrontThreads / 32;
    const T *gd = slab + S.blk_off[S.diag_pos[k]];
    if (tid == 0)
        s_extreme = 0;
    for (int c0 = 0; c0 < rows; c0 += 64)
        front_load(d + c0, ldd, gd + c0, m, m, m - c0, rows, min(64, rows - c0), warp, nw);
    front_load(b, kLdStrip, slab + S.blk_off[blk] + col0, K, m, w, rows, 8 * nb, warp, nw);
    __syncthreads();
    if (tid < m)
    {
        const double p = d[tid * ldd + tid];
        rpiv[tid] = front_reciprocal(p);
        if (front_extreme(p))
            s_extreme = 1;
    }
    __syncthreads();
    for (int r0 = 0; r0 < m; r0 += kPanel)
    {
        if (tid < 8 * nb)
            front_forward(d + r0 * ldd + r0, ldd, b + r0 * kLdStrip + tid, kLdStrip);
        __syncthreads();
        const int r1 = r0 + kPanel;
        for (int t = warp; t < nb * ((rows - r1 + 31) / 32); t += nw)
        {
            const int c0 = 8 * (t % nb), row = r1 + t / nb * 32;
            front_tiles<4>(b + c0, kLdStrip, d + r0, ldd, b + r0 * kLdStrip + c0, kLdStrip, row, min(row + 32, rows));
        }
        __syncthreads();
    }
    front_back(d, ldd, m, b, nb, rpiv, s_extreme != 0);
    T *out = wbuf + S.w_out[blockIdx.x] + col0;
    for (int r = warp; r < m; r += nw)
        for (int c = lane; c < w; c += 32)
            out[(int64_t)r * K + c] = (T)b[r * kLdStrip + c];
}

} // namespace hyb
