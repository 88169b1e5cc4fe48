// Panel factorisation of the FP64 LU with row partial pivoting (Simulation::solve_system with
// set_bcgstab(false): Eigen's PartialPivLU, Simulation.cpp:57-60), spread over the SMs.
//
// The right-looking blocked LU in linalg.cu factors each panel of nb columns (rows k0..n-1) and then
// updates the trailing matrix.  Each pivot decision needs the whole column, so a panel takes nb
// steps that each see all rows.  Here the panel's rows are split over G co-resident CTAs (one
// cooperative launch per panel), each holding its rows of the nb panel columns in shared memory for
// the whole panel.  A column step is one grid barrier:
//   * every CTA finds its largest |entry| of column j among its rows at or below the diagonal
//     (first row on ties) and publishes it with the full candidate row; the owner of the diagonal row
//     publishes that row too (double-buffered by column parity, so the next step's writes never meet
//     this step's reads);
//   * after the barrier every CTA picks the same pivot from the candidates in CTA order (largest
//     |entry|, then smallest row: the single-CTA kernel's rule), the owners of the two rows exchange
//     them, and every CTA eliminates below the diagonal with the pivot row: l = a_ij / a_jj,
//     a_ik -= l * a_jk for the panel columns right of j (the arithmetic of the single-CTA kernel).
// At the end each CTA writes its rows back.  A barrier wait that expires sets an error word; the
// caller then factors the matrix again with the single-CTA panel.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "ctx.h"
#include "grid_barrier.cuh"

namespace bemb {

namespace {

constexpr int LP_THREADS = 256;
constexpr int LP_NBMAX = 64;    // widest panel
constexpr int LP_GMAX = 1024;   // most CTAs of one panel

struct LPArgs {
    int n, k0, nb, rows_per;
    double* A;       // column-major n x n, factored in place
    int* piv;        // n: row interchanged with row k at step k
    int* sing;       // set on a zero pivot
    double* cand;    // 2 (parity) x G x (2 + nb): |entry|, row index, candidate row
    double* diag;    // 2 (parity) x nb: the diagonal row before the interchange
    unsigned* bar;   // grid barrier words
    int* err;        // barrier wait expired
    long long wait_limit;  // bound of each barrier wait, SM clock cycles
};

__global__ void __launch_bounds__(LP_THREADS) k_lu_panel_rows(LPArgs a) {
    extern __shared__ double sp[];  // [rows][ld], row-major; ld = nb + 1 (odd: no bank conflicts down a column)
    __shared__ double s_v[LP_THREADS / 32];
    __shared__ int s_i[LP_THREADS / 32];
    __shared__ int s_w[LP_THREADS / 32];
    __shared__ double s_prow[LP_NBMAX];
    const int n = a.n, nb = a.nb, G = gridDim.x, tid = threadIdx.x;
    const int r0 = a.k0 + blockIdx.x * a.rows_per, r1 = min(n, r0 + a.rows_per);
    const int nr = max(0, r1 - r0);
    const int stride = 2 + nb, ld = nb + 1;
    for (int e = tid; e < nr * nb; e += LP_THREADS) {
        const int c = e / nr, rr = e - c * nr;
        sp[rr * ld + c] = a.A[(size_t)(a.k0 + c) * n + r0 + rr];
    }
    __syncthreads();
    for (int j = 0; j < nb; ++j) {
        const int rowj = a.k0 + j;
        const int par = j & 1;
        double* cand = a.cand + (size_t)par * G * stride;
        double* diag = a.diag + (size_t)par * nb;
        // local pivot candidate: largest |a_ij| over owned rows i >= rowj, first row on ties
        double best = -1.0;
        int bi = n;
        for (int rr = tid; rr < nr; rr += LP_THREADS) {
            const int i = r0 + rr;
            if (i < rowj) continue;
            const double v = fabs(sp[rr * ld + j]);
            if (v > best || (v == best && i < bi)) {
                best = v;
                bi = i;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if ((tid & 31) == 0) {
            s_v[tid >> 5] = best;
            s_i[tid >> 5] = bi;
        }
        __syncthreads();
        if (tid < 32) {
            best = tid < LP_THREADS / 32 ? s_v[tid] : -2.0;
            bi = tid < LP_THREADS / 32 ? s_i[tid] : n;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) {
                    best = ov;
                    bi = oi;
                }
            }
            if (tid == 0) {
                s_v[0] = best;
                s_i[0] = bi;
            }
        }
        __syncthreads();
        best = s_v[0];
        bi = s_i[0];
        double* mine = cand + (size_t)blockIdx.x * stride;
        if (tid == 0) {
            mine[0] = best;
            mine[1] = (double)bi;
        }
        if (bi < n)
            for (int c = tid; c < nb; c += LP_THREADS) mine[2 + c] = sp[(bi - r0) * ld + c];
        if (rowj >= r0 && rowj < r1)
            for (int c = tid; c < nb; c += LP_THREADS) diag[c] = sp[(rowj - r0) * ld + c];
        if (!grid_barrier(a.bar, a.bar + 1, a.err, a.wait_limit)) return;
        // the pivot, the same in every CTA: largest |entry| over the candidates, then smallest row (an
        // order-independent rule, reduced over the threads)
        double pv = -1.0;
        int p = n, w = -1;
        for (int g = tid; g < G; g += LP_THREADS) {
            const double v = __ldcg(cand + (size_t)g * stride);
            const int i = (int)__ldcg(cand + (size_t)g * stride + 1);
            if (i < n && (v > pv || (v == pv && i < p))) {
                pv = v;
                p = i;
                w = g;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, pv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, p, o);
            const int ow = __shfl_xor_sync(0xffffffffu, w, o);
            if (oi < n && (ov > pv || (ov == pv && oi < p))) {
                pv = ov;
                p = oi;
                w = ow;
            }
        }
        if ((tid & 31) == 0) {
            s_v[tid >> 5] = pv;
            s_i[tid >> 5] = p;
            s_w[tid >> 5] = w;
        }
        __syncthreads();
        if (tid < 32) {
            pv = tid < LP_THREADS / 32 ? s_v[tid] : -1.0;
            p = tid < LP_THREADS / 32 ? s_i[tid] : n;
            w = tid < LP_THREADS / 32 ? s_w[tid] : -1;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, pv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, p, o);
                const int ow = __shfl_xor_sync(0xffffffffu, w, o);
                if (oi < n && (ov > pv || (ov == pv && oi < p))) {
                    pv = ov;
                    p = oi;
                    w = ow;
                }
            }
            if (tid == 0) {
                s_i[0] = p;
                s_w[0] = w;
            }
        }
        __syncthreads();
        p = s_i[0];
        w = s_w[0];
        if (p >= n) p = rowj;  // no candidate: keep the diagonal row
        const double* prow = (w >= 0) ? cand + (size_t)w * stride + 2 : diag;
        for (int c = tid; c < nb; c += LP_THREADS) s_prow[c] = __ldcg(prow + c);
        if (blockIdx.x == 0 && tid == 0) a.piv[rowj] = p;
        __syncthreads();
        // interchange: the pivot row goes to rowj, the old diagonal row to p
        if (p != rowj) {
            if (rowj >= r0 && rowj < r1)
                for (int c = tid; c < nb; c += LP_THREADS) sp[(rowj - r0) * ld + c] = s_prow[c];
            if (p >= r0 && p < r1)
                for (int c = tid; c < nb; c += LP_THREADS) sp[(p - r0) * ld + c] = __ldcg(diag + c);
        }
        __syncthreads();
        // eliminate below the diagonal with the pivot row
        const double d = s_prow[j];
        if (d == 0.0) {
            if (blockIdx.x == 0 && tid == 0) *a.sing = 1;
        }
        for (int rr = tid; rr < nr; rr += LP_THREADS) {
            const int i = r0 + rr;
            if (i <= rowj) continue;
            double l = sp[rr * ld + j];
            if (d != 0.0) {
                l /= d;
                sp[rr * ld + j] = l;
            }
            for (int c = j + 1; c < nb; ++c) sp[rr * ld + c] -= l * s_prow[c];
        }
        __syncthreads();
    }
    for (int e = tid; e < nr * nb; e += LP_THREADS) {
        const int c = e / nr, rr = e - c * nr;
        a.A[(size_t)(a.k0 + c) * n + r0 + rr] = sp[rr * ld + c];
    }
}

// One warp: tab_r[q] is a touched row, tab_s[q] the source row whose entries now sit there (both in
// shared memory, at most 2 nb entries).  Each transposition swaps the sources of its two rows; the
// lanes look a row up in parallel.  pairs[0] = m, then m (destination, source) pairs.
// A transposition whose partner row is not in (k0 + j, n) is skipped: it can only come from a panel
// whose bounded wait expired (an error the host reports), and skipping keeps every access in bounds.
__device__ void lu_build_pairs_warp(int n, int k0, int nb, const int* pj, int* tab_r, int* tab_s, int* pairs) {
    const int lane = threadIdx.x & 31;
    int cnt = 0;
    auto slot = [&](int r) {
        int found = -1;
        for (int q0 = 0; q0 < cnt && found < 0; q0 += 32) {
            const unsigned m = __ballot_sync(0xffffffffu, q0 + lane < cnt && tab_r[q0 + lane] == r);
            if (m) found = q0 + __ffs(m) - 1;
        }
        if (found >= 0) return found;
        if (lane == 0) {
            tab_r[cnt] = r;
            tab_s[cnt] = r;
        }
        __syncwarp();
        return cnt++;
    };
    for (int j = 0; j < nb; ++j) {
        const int rj = k0 + j, p = pj[j];
        if (p <= rj || p >= n) continue;
        const int a = slot(rj), b = slot(p);
        if (lane == 0) {
            const int t = tab_s[a];
            tab_s[a] = tab_s[b];
            tab_s[b] = t;
        }
        __syncwarp();
    }
    int m = 0;
    for (int q0 = 0; q0 < cnt; q0 += 32) {
        const int q = q0 + lane;
        const bool moved = q < cnt && tab_s[q] != tab_r[q];
        const unsigned bal = __ballot_sync(0xffffffffu, moved);
        if (moved) {
            const int k = m + __popc(bal & ((1u << lane) - 1u));
            pairs[1 + 2 * k] = tab_r[q];
            pairs[2 + 2 * k] = tab_s[q];
        }
        m += __popc(bal);
    }
    if (lane == 0) pairs[0] = m;
}

// The same panel on one thread-block cluster (up to 16 CTAs), for panels whose rows fit in the
// cluster's shared memory (about 6300 rows of a 64-column panel).  A thread owns one row: the row sits in
// shared memory, its entries in the current block of 8 columns in registers.  A column step is
//   * the largest |entry| of the column over the CTA's rows: one integer warp reduction of the high
//     words (and of the low words and rows on ties), one block barrier, one more warp reduction;
//   * every CTA sends its candidate (|entry|, row, reciprocal, the row's 8 block columns) into every
//     CTA's inbox through distributed shared memory, as 16-byte slots {value, step} written and read as
//     one access: no fence, no arrival, no second barrier.  Every warp polls (bounded) the inbox of its
//     own CTA and picks the pivot: largest |entry|, then smallest row;
//   * each thread eliminates its row in the block's registers, l = a_ij * (1 / a_jj), a_ik -= l a_jk.
// Rows are not moved: each thread keeps its row's position under the interchanges so far, and writes it
// there at the end.  The columns right of the block are updated once per block with rank 8, from the
// pivot rows' entries that their owner sent while the next candidates travelled.  Each entry sees the
// operations of the column-by-column elimination in the same order.
// Inboxes alternate by column parity: a CTA sends column j + 2's candidate only after it has read every
// CTA's for column j + 1, each sent after a block barrier behind the reads of column j.
// What bounds it: the serial chain of a column step, about 2500 cycles (reductions, barrier, a division,
// one distributed-shared-memory trip, the share of the rank-8 update).  Measured, mean over a solve's
// panels: 210 -> 94 us at N = 4002 and 172 -> 84 us at N = 984, against an exchange through mbarrier
// arrivals and fences by one warp, with the rows interchanged and all columns right of the current one
// updated in shared memory at every step.
// A wait that runs out sets *err; the CTA then takes what it finds, makes every send of the remaining
// columns (so no other CTA waits on it), and the caller factors again without the cluster.
constexpr int LC_MAX = 16;
constexpr size_t LC_SMEM = 220 * 1024;  // dynamic shared memory of one cluster CTA, at most
constexpr int LC_W = 8;                 // columns of a block
constexpr int LC_SLOTS = 12;            // slots of a candidate: key, row, reciprocal, LC_W entries, pad
constexpr int LC_REST = LP_NBMAX - LC_W;

__device__ __forceinline__ uint32_t lp_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16-byte slot {value, tag} of a CTA's shared memory (a cluster address), one access.
__device__ __forceinline__ void lc_send(uint32_t addr, unsigned long long v, unsigned long long tag) {
    asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.cluster.shared::cluster.b128 [%0], q;\n\t}" ::"r"(
                     addr),
                 "l"(v), "l"(tag)
                 : "memory");
}
__device__ __forceinline__ void lc_read(uint32_t addr, unsigned long long& v, unsigned long long& tag) {
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.cluster.shared::cta.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(v), "=l"(tag)
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ uint32_t lc_map(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// Lane of the largest key, of the smallest row among equal keys.
__device__ __forceinline__ int lc_argmax(unsigned long long key, int row) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    unsigned m;
    asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(m) : "r"(hi));
    bool in = hi == m;
    unsigned bal = __ballot_sync(0xffffffffu, in);
    if (bal & (bal - 1)) {
        asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(m) : "r"(in ? lo : 0u));
        in = in && lo == m;
        bal = __ballot_sync(0xffffffffu, in);
        if (bal & (bal - 1)) {
            int r;
            asm volatile("redux.sync.min.s32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(in ? row : 0x7fffffff));
            bal = __ballot_sync(0xffffffffu, in && row == r);
        }
    }
    return __ffs(bal) - 1;
}

// pairs (may be null): receives the panel's interchanges as (destination, source) row pairs.
template <int T>
__global__ void __launch_bounds__(T) k_lu_panel_cluster(int n, int k0, int nb, int rows_per, double* A, int* piv,
                                                        int* sing, int* pairs, int* err, long long wait_limit) {
    namespace cgx = cooperative_groups;
    using u64 = unsigned long long;
    cgx::cluster_group cl = cgx::this_cluster();
    constexpr int NW = T / 32, W = LC_W;
    // dynamic: inbox [2][C][LC_SLOTS], pivot rows [W][LC_REST] as slots; candidates of the warps
    // [2][NW][LC_SLOTS]; solved pivot rows [LC_REST][W]; multipliers of the pivot rows [W][W]; the rows
    extern __shared__ __align__(16) unsigned char sraw[];
    const int C = (int)cl.num_blocks(), me = (int)cl.block_rank(), tid = threadIdx.x;
    const int lane = tid & 31, wid = tid >> 5;
    const int ld = nb | 1;
    ulonglong2* inbox = reinterpret_cast<ulonglong2*>(sraw);
    ulonglong2* ubox = inbox + 2 * C * LC_SLOTS;
    u64* cand = reinterpret_cast<u64*>(ubox + W * LC_REST);
    double* usol = reinterpret_cast<double*>(cand + 2 * NW * LC_SLOTS);
    double* pl = usol + LC_REST * W;
    double* sp = pl + W * W;
    const int r0 = k0 + me * rows_per, nr = max(0, min(n, r0 + rows_per) - r0);
    const uint32_t inbox_a = lp_smem(inbox), ubox_a = lp_smem(ubox);
    for (int e = tid; e < 2 * C * LC_SLOTS + W * LC_REST; e += T) inbox[e] = make_ulonglong2(0, 0);
    if (pairs && me == 0 && tid == 0) pairs[0] = 0;
    const bool valid = tid < nr;
    double* row = sp + (size_t)tid * ld;
    if (valid)
        for (int c0 = 0; c0 < nb; c0 += 16) {  // 16 loads in flight
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = c0 + u < nb ? A[(size_t)(k0 + c0 + u) * n + r0 + tid] : 0.0;
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (c0 + u < nb) row[c0 + u] = v[u];
        }
    cl.sync();  // every CTA's slots are clear before anyone writes into them
    int pos = valid ? r0 + tid : 0x7fffffff;  // the row's position after the interchanges so far
    bool active = valid, ok = true;
    int send_k = -1, send_row = 0;  // the last column's pivot row, if this CTA's: its block step and row
    for (int jb = 0; jb < nb; jb += W) {
        const int rest = nb - jb - W;  // columns right of the block
        double v[W];
#pragma unroll
        for (int c = 0; c < W; ++c) v[c] = valid && jb + c < nb ? row[jb + c] : 0.0;
        int kd = -1;  // the block step at which this row became a pivot row
        // the pivot row of step send_k goes to every CTA, its entries right of the block
        auto send_pivot_row = [&]() {
            if (send_k < 0) return;
            for (int d = wid; d < C; d += NW) {
                const uint32_t to = lc_map(ubox_a, d) + send_k * LC_REST * 16;
                for (int c = lane; c < rest; c += 32)
                    lc_send(to + c * 16, __double_as_longlong(sp[(size_t)send_row * ld + jb + W + c]), jb + send_k + 1);
            }
            send_k = -1;
        };
#pragma unroll
        for (int jj = 0; jj < W; ++jj) {
            const int j = jb + jj;
            if (j >= nb) break;
            const int rowj = k0 + j, par = j & 1;
            const u64 tag = j + 1;
            u64* mine = cand + (size_t)(par * NW + wid) * LC_SLOTS;
            // |entry| as an integer, ordered like the value; a NaN is below every number
            const double av = fabs(v[jj]);
            u64 key = active && av == av ? (u64)__double_as_longlong(av) + 1 : 0;
            int kr = active ? pos : 0x7fffffff;
            const int wl = lc_argmax(key, kr);
            if (lane == wl) {
                mine[0] = key;
                mine[1] = (u64)(unsigned)kr | (u64)(unsigned)tid << 32;
                mine[2] = __double_as_longlong(v[jj] != 0.0 ? 1.0 / v[jj] : 0.0);
#pragma unroll
                for (int c = 0; c < W; ++c) mine[3 + c] = __double_as_longlong(v[c]);
            }
            __syncthreads();
            const u64* wc = cand + (size_t)par * NW * LC_SLOTS;
            key = lane < NW ? wc[lane * LC_SLOTS] : 0;
            kr = lane < NW ? (int)wc[lane * LC_SLOTS + 1] : 0x7fffffff;
            const int ww = lc_argmax(key, kr);
            const int dest = wid + (lane >> 4) * NW, sl = lane & 15;
            if (dest < C && sl < 3 + W)
                lc_send(lc_map(inbox_a, dest) + ((par * C + me) * LC_SLOTS + sl) * 16, wc[ww * LC_SLOTS + sl], tag);
            send_pivot_row();
            // every CTA's candidate
            const uint32_t box = inbox_a + par * C * LC_SLOTS * 16;
            u64 a0 = 0, a1 = 0x7fffffff, t0, t1;
            long long tw = 0;
            for (;;) {
                bool have = true;
                if (lane < C) {
                    lc_read(box + lane * LC_SLOTS * 16, a0, t0);
                    lc_read(box + lane * LC_SLOTS * 16 + 16, a1, t1);
                    have = t0 == tag && t1 == tag;
                }
                if (__all_sync(0xffffffffu, have)) break;
                const long long now = clock64();
                if (!tw) tw = now;
                if (__any_sync(0xffffffffu, !ok || now - tw >= wait_limit)) {
                    ok = false;
                    if (!have) {
                        a0 = 0;
                        a1 = 0x7fffffff;
                    }
                    break;
                }
            }
            const int w = lc_argmax(a0, (int)a1);
            int p = (int)__shfl_sync(0xffffffffu, (unsigned)a1, w);
            const int prow = (int)__shfl_sync(0xffffffffu, (unsigned)(a1 >> 32), w);
            if (p < rowj || p >= n) {  // only after an expired wait: keep every index in range
                p = rowj;
                ok = false;
            }
            // its reciprocal and block entries, and (warp 0) its earlier multipliers for the rank-8 update
            double u[W], rcp;
            const uint32_t ws = box + min(w, C - 1) * LC_SLOTS * 16;
            for (;;) {
                u64 tags[W + 1], x;
                lc_read(ws + 32, x, tags[W]);
                rcp = __longlong_as_double(x);
                bool have = tags[W] == tag;
#pragma unroll
                for (int c = 0; c < W; ++c) {
                    lc_read(ws + 48 + c * 16, x, tags[c]);
                    u[c] = __longlong_as_double(x);
                    have = have && tags[c] == tag;
                }
                if (have || !ok) break;
                const long long now = clock64();
                if (!tw) tw = now;
                if (now - tw >= wait_limit) ok = false;
            }
            if (tid == 0) {
#pragma unroll
                for (int c = 0; c < jj; ++c) pl[jj * W + c] = u[c];
                if (me == 0) {
                    piv[rowj] = p;
                    if (u[jj] == 0.0) *sing = 1;
                }
            }
            if (active) {
                if (pos == p) {
                    active = false;
                    kd = jj;
                    pos = rowj;
                } else {
                    if (pos == rowj) pos = p;
                    double l = v[jj];
                    if (rcp != 0.0) l *= rcp;
                    v[jj] = l;
#pragma unroll
                    for (int c = jj + 1; c < W; ++c) v[c] -= l * u[c];
                }
            }
            if (w == me && rest > 0) {
                send_k = jj;
                send_row = min(prow, nr - 1);
            }
        }
        if (valid && (active || kd >= 0)) {
#pragma unroll
            for (int c = 0; c < W; ++c)
                if (jb + c < nb) row[jb + c] = v[c];
        }
        if (rest <= 0) continue;
        send_pivot_row();
        __syncthreads();  // the pivot rows' multipliers
        if (tid < rest) {
            // column jb + W + tid of the block's pivot rows, each less the pivot rows before it
            double u[W];
            long long tw = 0;
            for (;;) {
                bool have = true;
#pragma unroll
                for (int k = 0; k < W; ++k) {
                    u64 x, t;
                    lc_read(ubox_a + (k * LC_REST + tid) * 16, x, t);
                    u[k] = __longlong_as_double(x);
                    have = have && t == (u64)(jb + k + 1);
                }
                if (have || !ok) break;
                const long long now = clock64();
                if (!tw) tw = now;
                if (now - tw >= wait_limit) ok = false;
            }
#pragma unroll
            for (int k = 0; k < W; ++k) {
#pragma unroll
                for (int i = 0; i < k; ++i) u[k] -= pl[k * W + i] * u[i];
                usol[tid * W + k] = u[k];
            }
        }
        __syncthreads();
        if (active) {
#pragma unroll 4
            for (int c = 0; c < rest; ++c) {
                double x = row[jb + W + c];
#pragma unroll
                for (int k = 0; k < W; ++k) x -= v[k] * usol[c * W + k];
                row[jb + W + c] = x;
            }
        } else if (kd >= 0) {
            for (int c = 0; c < rest; ++c) row[jb + W + c] = usol[c * W + kd];
        }
    }
    if (__any_sync(0xffffffffu, !ok) && lane == 0) atomicExch(err, 1);
    cl.sync();  // no CTA leaves while another may still write into its shared memory
    if (valid && pos < n) {
        for (int c = 0; c < nb; ++c) A[(size_t)(k0 + c) * n + pos] = row[c];
        if (pairs && pos != r0 + tid) {
            const int k = atomicAdd(pairs, 1);
            if (k < 2 * LP_NBMAX) {
                pairs[1 + 2 * k] = pos;
                pairs[2 + 2 * k] = r0 + tid;
            }
        }
    }
}

// The panel's transpositions (k0 + j, pj[j]) composed into (destination, source) row pairs by one warp;
// k_lu_swap_trsm (linalg.cu) applies them.
__global__ void __launch_bounds__(32) k_lu_perm_build(int n, int k0, int nb, const int* __restrict__ piv,
                                                      int* __restrict__ pairs) {
    __shared__ int tab_r[2 * LP_NBMAX], tab_s[2 * LP_NBMAX];
    lu_build_pairs_warp(n, k0, nb, piv + k0, tab_r, tab_s, pairs);
}

}  // namespace

// lu_aux layout: candidates (2 parities x LP_GMAX x (2 + nb)), diagonal rows (2 x LP_NBMAX),
// barrier words (2), error word
static double* lp_diag(Ctx& c) { return c.lu_aux + (size_t)2 * LP_GMAX * (2 + LP_NBMAX); }
static unsigned* lp_bar(Ctx& c) { return reinterpret_cast<unsigned*>(lp_diag(c) + 2 * LP_NBMAX); }

// then the interchange pairs of the last panel (1 + 2 x 2 LP_NBMAX ints)
static int* lp_pairs(Ctx& c) { return reinterpret_cast<int*>(lp_bar(c) + 4); }

size_t lu_panel_words() { return (size_t)2 * LP_GMAX * (2 + LP_NBMAX) + (size_t)2 * LP_NBMAX + 8 + 2 * LP_NBMAX + 8; }

const int* lu_panel_pairs(Ctx& c, int k0, int nb, cudaStream_t s, bool built) {
    const int n = (int)c.topo.N;
    if (!built) KLAUNCH(), k_lu_perm_build<<<1, 32, 0, s>>>(n, k0, nb, c.piv, lp_pairs(c));
    return lp_pairs(c);
}

template <int T>
static int launch_panel_cluster(Ctx& c, int n, int k0, int nb, int C, int rows_per, double* A, int* piv, int* sing,
                                bool want_pairs, cudaStream_t s) {
    const size_t smem = 16 * ((size_t)2 * C * LC_SLOTS + LC_W * LC_REST) +
                        8 * ((size_t)2 * (T / 32) * LC_SLOTS + LC_REST * LC_W + LC_W * LC_W + (size_t)rows_per * (nb | 1));
    if (smem > LC_SMEM) return BEM_ERR_CUDA;
    static std::atomic<uint64_t> attr{0};
    if (!once_per_device(attr, [] {
            return cudaFuncSetAttribute(k_lu_panel_cluster<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)LC_SMEM) == cudaSuccess &&
                   cudaFuncSetAttribute(k_lu_panel_cluster<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                       cudaSuccess;
        })) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_lu_panel_cluster<T>, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    KLAUNCH();
    int* pairs = want_pairs ? lp_pairs(c) : nullptr;  // the interchange pairs of c.LU's panel
    if (cudaLaunchKernelEx(&cfg, k_lu_panel_cluster<T>, n, k0, nb, rows_per, A, piv, sing, pairs, lu_panel_err(c),
                           (long long)c.wait_limit) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    return BEM_OK;
}

// The panel on one thread-block cluster when its rows fit; BEM_ERR_CUDA when they do not or the
// cluster launch is unavailable.
int lu_panel_cluster(Ctx& c, int k0, int nb, cudaStream_t s, const PanelTarget* tgt) {
    const int n = tgt ? tgt->n : (int)c.topo.N;
    double* A = tgt ? tgt->A : c.LU;
    int* piv = tgt ? tgt->piv : c.piv;
    int* sing = tgt ? tgt->sing : c.flag;
    const int P = n - k0;
    if (nb > LP_NBMAX) return BEM_ERR_CUDA;
    // one row per thread; as few CTAs as hold the rows with 256 threads each (512 above 16 x 256 rows):
    // the exchange's cost grows little with the CTAs, but none of them does any work in it
    const int C = std::max(1, std::min(LC_MAX, (P + 255) / 256));
    const int rows_per = (P + C - 1) / C;
    if (rows_per > 512) return BEM_ERR_CUDA;
    return rows_per <= 256 ? launch_panel_cluster<256>(c, n, k0, nb, C, rows_per, A, piv, sing, tgt == nullptr, s)
                           : launch_panel_cluster<512>(c, n, k0, nb, C, rows_per, A, piv, sing, tgt == nullptr, s);
}

int* lu_panel_err(Ctx& c) { return reinterpret_cast<int*>(lp_bar(c) + 2); }

// Factor panel [k0, k0+nb) of c.LU (or of tgt's matrix) over rows k0..n-1.  Returns BEM_ERR_CUDA when the cooperative
// launch is unavailable or a barrier wait expired (the caller falls back to the single-CTA panel,
// from a fresh copy of the matrix).
int lu_panel_rows(Ctx& c, int k0, int nb, cudaStream_t s, const PanelTarget* tgt) {
    const int n = tgt ? tgt->n : (int)c.topo.N;
    int sms = 0, coop = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device);
    if (!coop) return BEM_ERR_CUDA;
    const int P = n - k0;
    const int G = std::max(1, std::min(sms, (P + 127) / 128));
    const int rows_per = (P + G - 1) / G;
    if (nb > LP_NBMAX || G > LP_GMAX) return BEM_ERR_CUDA;
    const size_t smem = sizeof(double) * (size_t)rows_per * (nb + 1);
    if (smem > 200 * 1024) return BEM_ERR_CUDA;
    static std::atomic<uint64_t> attr{0};
    if (!once_per_device(attr, [] {
            return cudaFuncSetAttribute(k_lu_panel_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) ==
                   cudaSuccess;
        })) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lu_panel_rows, LP_THREADS, smem) != cudaSuccess ||
        per_sm * sms < G)
        return BEM_ERR_CUDA;
    LPArgs a{};
    a.n = n;
    a.k0 = k0;
    a.nb = nb;
    a.rows_per = rows_per;
    a.A = tgt ? tgt->A : c.LU;
    a.piv = tgt ? tgt->piv : c.piv;
    a.sing = tgt ? tgt->sing : c.flag;
    a.cand = c.lu_aux;
    a.diag = lp_diag(c);
    a.bar = lp_bar(c);
    a.err = lu_panel_err(c);  // cleared once per factorisation by the caller
    a.wait_limit = c.wait_limit;
    BEM_CUDA(c, cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned), s));
    void* args[] = {&a};
    KLAUNCH();
    cudaError_t e = cudaLaunchCooperativeKernel((void*)k_lu_panel_rows, G, LP_THREADS, args, smem, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    return BEM_OK;
}

}  // namespace bemb
