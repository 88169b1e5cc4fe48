// BiCGSTAB with the vectors resident on the SMs (the reference's default solver, Simulation.cpp:49-53:
// Jacobi preconditioner, zero start, tolerance DBL_EPSILON on the recursive residual, at most 2N
// iterations, shadow-residual restart): the whole solve in one cooperative launch, for N <= 6144.  Up to
// N = 2028 (32.9 MB) the matrix too stays in the register files and shared memories of the GPU; above, it is
// streamed from L2 and HBM.
//
// What bounds it, matrix resident: a product reads nothing from outside the SM and takes well under a
// microsecond, so an iteration costs its two all-to-all exchanges and the chain of dot products.
//   * A CTA owns 16 rows (or N / SMs, if that is more), a thread up to 28 entries of one row in
//     registers and the rest in shared memory.  Few CTAs: every CTA reads every published vector, and
//     with 16 rows the slots of a CTA fill whole 128-byte lines, which are polled by all the others.
//     Measured at N = 812, per iteration: 6.1 us with 16 rows, 7.0 with 8, 7.8 with 12 and 8.3 with 6
//     (one CTA per SM).
//   * Every CTA keeps all of r, p, v (in registers, the same elements in the same thread everywhere) and
//     updates them redundantly, in the same order, so every CTA holds the same bits and takes the same
//     decisions.  That leaves two exchanges per iteration (v = A y and t = A z) instead of the five
//     grid barriers of k_pbicg (bicg.cu).
//   * An exchange has no barrier: a published element is a 16-byte slot {value, sequence number}, written
//     and read as one 128-bit access, and a reader polls the slots it needs until they carry the current
//     number.  Two sets of slots by the number's parity suffice: a CTA publishes number s + 2 only after
//     it has read all of s + 1, which every other CTA published after it had read all of s.  Sequence
//     numbers grow over the context's solves, so the slots are cleared only when they are allocated.
//     1.3 to 1.8 us per exchange over 50 to 140 CTAs; a counter barrier and a read of the vector take
//     1.9 to 2.4 us.
// Measured (B200, whole solve, against k_pbicg in batches of 64 iterations): N = 162: 0.10 ms (0.63),
// N = 812 with the wall image: 0.23 ms (1.13), N = 1442: 0.35 ms (1.66), N = 1962: 0.54 ms.
//
// Matrix streamed: bound by the two reads of the matrix per iteration.  Each thread copies two rows of its
// columns (16 bytes) into a ring of its own in shared memory, 12 copies ahead in groups of four (98 KB in flight
// per SM, no registers held, no barrier: a thread reads only what it copied), and the copies run on through the
// exchanges.  One copy per group took 1 to 3 % longer up to N = 4096.
// 64 MB of the matrix are marked to stay in L2 (evict_last, the rest evict_first).  Per iteration: N = 4002:
// 38 us (6.7 TB/s of matrix reads) against 91 us for k_pbicg; 42 us without the marks, 47 us with 100 MB marked.
// With loads into registers instead of the ring 48 us; with a TMA ring of row slabs 71 us (a slab's rows are
// 224 bytes, too short for the copy engine).  N = 2562: 24 us; N = 5762: 84 us.
//
// A wait is bounded (Ctx::wait_limit): a warp that gives up sets the error word and its CTA returns; the
// others then run out of their own waits.  The host finishes the solve with the multi-kernel form.
#include <math.h>

#include <algorithm>
#include <cmath>

#include "ctx.h"
#include "resident.cuh"

namespace bemb {

namespace {

constexpr int RB_U = 4;                // streamed: columns per group of copies
constexpr int RB_D8 = 12, RB_D12 = 8;  // streamed: copies in flight per thread, up to 4096 and 6144 unknowns
constexpr double RB_EPS = 2.220446049250313080847e-16;

struct RBArgs {
    int n, ld, rows, nv, npart, maxit;  // rows per CTA; doubles of the input vector and of the row partials
    int nk;                            // streamed: groups of RB_U columns per thread
    float keep;                        // streamed: share of the matrix to keep in L2
    const double* A;
    const double* b;
    double* x;
    ulonglong2* ex;            // 2 x n exchange slots {value, sequence number}
    unsigned long long seq;    // sequence numbers of this solve start above this
    DevScalars* sc;            // results: iterations, residual norms, convergence; the error word
    long long wait_limit;      // bound of each exchange wait, SM clock cycles
};

enum { PH_V, PH_T, PH_RX, PH_RT };

// D > 0: the matrix is streamed, D copies in flight per thread; D = 0: it is resident, M entries per thread in
// registers and the rest in shared memory.
template <int K, int M, int D>
__global__ void __launch_bounds__(RB_T, 1) k_bicg_resident(const RBArgs a) {
    constexpr bool ST = D > 0;
    extern __shared__ __align__(16) double smem[];
    const int n = a.n, np = (n + 1) & ~1, nv = a.nv, tid = threadIdx.x, rows = a.rows;
    const int row0 = blockIdx.x * rows, nr = min(rows, n - row0);
    const int per = ST ? rows / 2 : rows, cstep = RB_T / per;  // threads down a column, columns side by side
    // streamed: the ring; the input vector, shadow residual and Jacobi diagonal; row partials; sums; the slab
    double2* ring = reinterpret_cast<double2*>(smem) + tid;  // slot d at d RB_T
    double* vec = smem + (size_t)2 * D * RB_T;
    double *r0 = vec + nv, *invd = r0 + np, *part = invd + np, *red = part + a.npart;
    double* slab = red + 6 * RB_WARPS;
    const int i = tid % per * (ST ? 2 : 1), c = tid / per;  // the thread's (first) row of the CTA, first column
    const bool active = c < cstep && i < nr;
    // the stream of a thread: its two rows of columns c, c + cstep, ..., product after product
    uint64_t pol = 0;
    const double* next = a.A + (size_t)min(c, n - 1) * a.ld + row0 + min(i, nr - 1);
    int nextj = c, slot = 0;
    auto advance = [&](int d) {
#pragma unroll
        for (int u = 0; u < RB_U; ++u)
            if (active) ring_copy(ring + (d + u) * RB_T, next + (size_t)u * cstep * a.ld, nextj + u * cstep < n, pol);
        asm volatile("cp.async.commit_group;" ::: "memory");
        nextj += RB_U * cstep;
        next += (size_t)RB_U * cstep * a.ld;
        if (nextj >= a.nk * RB_U * cstep) {  // the next product
            nextj -= a.nk * RB_U * cstep;
            next -= (size_t)a.nk * RB_U * cstep * a.ld;
        }
    };
    if (ST) {
        asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, %1;" : "=l"(pol) : "f"(a.keep));
#pragma unroll
        for (int d = 0; d < D; d += RB_U) advance(d);
    }
    // the thread's entries of the own rows (not ST): columns c + q cstep, the first M in registers, the others
    // (columns from M cstep on) in shared memory
    double m[M ? M : 1];
#pragma unroll
    for (int q = 0; q < M; ++q) {
        const int j = c + q * cstep;
        m[q] = active && j < n ? __ldg(a.A + (size_t)j * a.ld + row0 + i) : 0.0;
    }
    if (!ST && active)
        for (int j = c + M * cstep; j < n; j += cstep)
            slab[(j - M * cstep) * rows + i] = __ldg(a.A + (size_t)j * a.ld + row0 + i);
    for (int e = n + tid; e < nv; e += RB_T) vec[e] = 0.0;  // read with the zero entries past column n
    // r (s between the two products), p (p - w v after the second), v of the thread's elements
    double r[K], p[K], v[K];
    double bb = 0.0, dummy;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int e = tid + k * RB_T;
        r[k] = p[k] = v[k] = 0.0;
        if (e < n) {
            const double d = __ldg(a.A + (size_t)e * a.ld + e), be = __ldg(a.b + e);
            invd[e] = d != 0.0 ? 1.0 / d : 1.0;
            r0[e] = be;
            r[k] = be;
            bb += be * be;
        }
    }
    cta_sums(red + 4 * RB_WARPS, bb, 0.0, true, bb, dummy);
    const double tol2 = RB_EPS * RB_EPS * bb;
    double rr = bb, r0r = bb, r0_sq = bb, rho = 1.0, alpha = 1.0, w = 1.0;
    double bfac = 1.0;  // (alpha / w) / rho of the iteration before: beta = rho bfac
    double x = 0.0, y = 0.0;  // of row row0 + tid, tid < nr
    int iters = 0, restarts = 0, nonconv = 0, phase = PH_V;
    unsigned long long seq = a.seq;
    bool begin = bb != 0.0, go = begin;
    while (go) {
        if (begin) {  // a new iteration: loop test, then p and y = invd p, or a restart
            begin = false;
            if (!(rr > tol2) || iters >= a.maxit) {
                nonconv = rr > tol2 ? 1 : 0;
                break;
            }
            rho = r0r;
            phase = fabs(r0r) < RB_EPS * RB_EPS * r0_sq ? PH_RX : PH_V;
        }
        ++seq;
        ulonglong2* slots = a.ex + (size_t)(seq & 1) * n;
        if (phase == PH_RX) {  // the restart needs all of x
            if (tid < nr) slot_store(slots + row0 + tid, x, seq);
        } else {
            if (phase == PH_V) {
                const double beta = rho * bfac;
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (tid + k * RB_T < n) {
                        p[k] = r[k] + beta * p[k];
                        vec[tid + k * RB_T] = invd[tid + k * RB_T] * p[k];
                    }
            }
            __syncthreads();
            // the own rows of A vec
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            if (ST) {
                for (int k = 0; k < a.nk; ++k) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(ST ? D / RB_U - 1 : 0) : "memory");
                    const double* vc = vec + c + k * RB_U * cstep;
                    double2 v[RB_U];
                    double xv[RB_U];
#pragma unroll
                    for (int u = 0; u < RB_U; ++u) {
                        v[u] = ring[(slot + u) * RB_T];
                        xv[u] = vc[u * cstep];
                    }
#pragma unroll
                    for (int u = 0; u < RB_U; ++u) {
                        acc[0] = fma(v[u].x, xv[u], acc[0]);
                        acc[1] = fma(v[u].y, xv[u], acc[1]);
                    }
                    advance(slot);
                    slot = slot + RB_U == D ? 0 : slot + RB_U;
                }
                if (active) {
                    part[i * (cstep + 1) + c] = acc[0];
                    part[(i + 1) * (cstep + 1) + c] = acc[1];
                }
            } else if (active) {
                const double* vc = vec + c;
#pragma unroll
                for (int q = 0; q < M; ++q) acc[q & 3] = fma(m[q], vc[q * cstep], acc[q & 3]);
                int j = c + M * cstep;
                const double* sl = slab + c * rows + i;
                const int sst = cstep * rows;
                for (; j + 3 * cstep < n; j += 4 * cstep, sl += 4 * sst) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[q] = fma(sl[q * sst], vec[j + q * cstep], acc[q]);
                }
                for (; j < n; j += cstep, sl += sst) acc[0] = fma(sl[0], vec[j], acc[0]);
            }
            if (!ST && active) part[i * (cstep + 1) + c] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
            __syncthreads();
            const int lane = tid & 31;
            for (int q = tid >> 5; q < nr; q += RB_WARPS) {
                double s = 0.0;
                for (int k = lane; k < cstep; k += 32) s += part[q * (cstep + 1) + k];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) slot_store(slots + row0 + q, s, seq);
            }
            if (phase == PH_V && tid < nr) y = vec[row0 + tid];
        }
        double t[K];
        const bool ok = collect<K>(slots, n, seq, a.wait_limit, t);
        if (!ok && (tid & 31) == 0) atomicExch(&a.sc->wait_err, 1);
        if (phase == PH_V) {
            double s0 = 0.0, r0v;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                v[k] = t[k];
                if (tid + k * RB_T < n) s0 += r0[tid + k * RB_T] * v[k];
            }
            if (!cta_sums(red, s0, 0.0, ok, r0v, dummy)) break;
            alpha = rho / r0v;
            // s = r - alpha v; z = invd s
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (tid + k * RB_T < n) {
                    r[k] = r[k] - alpha * v[k];
                    vec[tid + k * RB_T] = invd[tid + k * RB_T] * r[k];
                }
            phase = PH_T;
        } else if (phase == PH_T) {
            const double z = tid < nr ? vec[row0 + tid] : 0.0;
            double s0 = 0.0, s1 = 0.0, tt, ts;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                s0 += t[k] * t[k];
                s1 += t[k] * r[k];
            }
            if (!cta_sums(red + 2 * RB_WARPS, s0, s1, ok, tt, ts)) break;
            w = tt > 0.0 ? ts / tt : 0.0;
            bfac = (alpha / w) / rho;
            x += alpha * y + w * z;
            s0 = s1 = 0.0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                r[k] = r[k] - w * t[k];
                p[k] = p[k] - w * v[k];
                s0 += r[k] * r[k];
                if (tid + k * RB_T < n) s1 += r0[tid + k * RB_T] * r[k];
            }
            cta_sums(red + 4 * RB_WARPS, s0, s1, true, rr, r0r);
            ++iters;
            begin = true;
        } else if (phase == PH_RX) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (tid + k * RB_T < n) vec[tid + k * RB_T] = t[k];
            if (__syncthreads_or(!ok)) break;
            phase = PH_RT;
        } else {  // r = b - A x, r0 = r
            double s0 = 0.0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int e = tid + k * RB_T;
                if (e < n) {
                    r[k] = __ldg(a.b + e) - t[k];
                    r0[e] = r[k];
                    s0 += r[k] * r[k];
                }
            }
            if (!cta_sums(red, s0, 0.0, ok, rho, dummy)) break;
            r0_sq = rho;
            if (restarts++ == 0) iters = 0;
            phase = PH_V;
        }
    }
    if (ST) asm volatile("cp.async.wait_all;" ::: "memory");
    if (tid < nr) a.x[row0 + tid] = x;
    if (blockIdx.x == 0 && tid == 0) {
        a.sc->rhs_sq = bb;
        a.sc->rr = rr;
        a.sc->iters = iters;
        a.sc->nonconv = nonconv;
        a.sc->done = 1;
    }
}

template <int K, int M, int D>
cudaError_t rb_launch(const RBArgs& a, int grid, size_t smem, cudaStream_t s) {
    static std::atomic<uint64_t> ready{0};
    if (!once_per_device(ready, [] {
            return cudaFuncSetAttribute(k_bicg_resident<K, M, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        RB_SMEM) == cudaSuccess;
        }))
        return cudaErrorUnknown;
    void* args[] = {const_cast<RBArgs*>(&a)};
    return cudaLaunchCooperativeKernel((void*)k_bicg_resident<K, M, D>, grid, RB_T, args, smem, s);
}

}  // namespace

size_t rbicg_words(int64_t n) { return n <= RB_MAX_N ? 4 * (size_t)n : 0; }

int bicgstab_resident(Ctx& c, const double* A, const double* b, double* x, cudaStream_t s) {
    const int n = (int)c.topo.N;
    const int maxit = c.prm.max_iters > 0 ? c.prm.max_iters : 2 * n;
    int sms = 0, coop = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device);
    if (!coop || n > RB_MAX_N || maxit > 4 * RB_MAX_N) return BEM_ERR_STATE;
    RBArgs a{};
    a.n = n;
    a.ld = n;
    a.maxit = maxit;
    a.b = b;
    a.x = x;
    a.ex = reinterpret_cast<ulonglong2*>(c.rbicg);
    a.sc = c.sc;
    a.wait_limit = c.wait_limit;
    const int np = (n + 1) & ~1, K = (n + RB_T - 1) / RB_T;
    int grid = 0;
    size_t smem = RB_SMEM + 1;
    // the matrix on the SMs where a CTA's rows fit: on 148 of them 225.9 KB at N = 2028, 226.1 KB at 2029 (226 at
    // most); else streamed
    if (n <= RB_RES_N) {
        a.rows = std::max(std::min(n, 16), (n + sms - 1) / sms);
        grid = (n + a.rows - 1) / a.rows;
        const int cstep = RB_T / a.rows;
        const int M = K == 1 ? (n <= 8 * cstep ? 8 : 16) : K == 2 ? 28 : K == 3 ? 24 : 20;
        a.nv = std::max(np, M * cstep);
        a.nv += a.nv & 1;
        a.npart = a.rows * (cstep + 1);
        smem = sizeof(double) *
               (a.nv + 2 * (size_t)np + a.npart + 6 * RB_WARPS + (size_t)std::max(0, n - M * cstep) * a.rows);
    }
    const bool stream = smem > RB_SMEM;
    if (stream) {
        a.rows = ((n + sms - 1) / sms + 1) & ~1;  // even: a copy takes two rows
        grid = (n + a.rows - 1) / a.rows;
        const int cstep = RB_T / (a.rows / 2), D = K <= 8 ? RB_D8 : RB_D12;
        a.nk = (n + RB_U * cstep - 1) / (RB_U * cstep);
        a.nv = (a.nk * RB_U * cstep + cstep + 1) & ~1;  // idle threads read a little past their columns
        a.npart = a.rows * (cstep + 1);
        smem = sizeof(double) * ((size_t)2 * D * RB_T + a.nv + 2 * (size_t)np + a.npart + 6 * RB_WARPS);
        if (smem > RB_SMEM || a.rows > 2 * RB_T || !c.LU) return BEM_ERR_STATE;
        // the part of the matrix that the L2 can hold beside the stream
        a.keep = (float)std::min(1.0, RB_KEEP / (8.0 * n * n));
        if (n % 2 || reinterpret_cast<uintptr_t>(A) % 16) {  // copies of 16 bytes: a matrix with an even stride
            a.ld = (n + 1) & ~1;
            BEM_CUDA(c, cudaMemcpy2DAsync(c.LU, sizeof(double) * a.ld, A, sizeof(double) * n, sizeof(double) * n, n,
                                          cudaMemcpyDeviceToDevice, s));
            A = c.LU;
        }
    }
    a.A = A;
    a.seq = ++c.rbicg_solves << 32;
    KLAUNCH();
    const cudaError_t e = stream   ? (K <= 8 ? rb_launch<8, 0, RB_D8>(a, grid, smem, s)
                                             : rb_launch<12, 0, RB_D12>(a, grid, smem, s))
                          : K == 1 ? (n <= 8 * (RB_T / a.rows) ? rb_launch<1, 8, 0>(a, grid, smem, s)
                                                               : rb_launch<1, 16, 0>(a, grid, smem, s))
                          : K == 2 ? rb_launch<2, 28, 0>(a, grid, smem, s)
                          : K == 3 ? rb_launch<3, 24, 0>(a, grid, smem, s)
                                   : rb_launch<4, 20, 0>(a, grid, smem, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    BEM_CUDA(c, cudaMemcpyAsync(c.h_sc, c.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s));
    BEM_CUDA(c, cudaStreamSynchronize(s));
    if (c.h_sc->wait_err) {
        BEM_CUDA(c, cudaMemsetAsync(&c.sc->wait_err, 0, sizeof(int32_t), s));
        c.stats.wait_expired++;
        return c.fail(BEM_ERR_CUDA, "BiCGSTAB: an exchange wait expired");
    }
    // (alpha / w) / rho, kept for the next beta, leaves the FP64 range where rho falls below 1e-308 (a b of norm 1e-148
    // or less); beta = (rho / rho_old) (alpha / w), as the other forms have it, does not
    if (!std::isfinite(c.h_sc->rr)) return BEM_ERR_STATE;
    c.stats.last_iters = c.h_sc->iters;
    c.stats.last_rel_residual = c.h_sc->rhs_sq > 0 ? sqrt(c.h_sc->rr / c.h_sc->rhs_sq) : 0.0;
    c.stats.total_iters += c.stats.last_iters;
    c.stats.solves++;
    return BEM_OK;
}

}  // namespace bemb
