// Iterative refinement x <- x + X (b - G x) of the mixed solver as one cooperative launch per round, for
// N <= 6144: the vectors on the SMs as in bicg_resident.cu, G (FP64) and the approximate inverse X (FP32)
// streamed from L2 and HBM, the convergence test on the device.
//
// What bounds it: the reads of G and X, 12 N^2 bytes per step.  As separate launches a step's two GEMVs each
// pay their ramp, the tail of the column splits and, at small sizes, mostly the launch; the number of steps had
// to be guessed, with gated extra steps behind it.  Here a thread copies 16 bytes (two rows of G or four of X)
// per column into a ring of its own, RF_D copies ahead across the products and exchanges, RB_KEEP bytes marked to
// stay in L2.  Two exchanges per step (bicg_resident.cu describes them).
// Measured (B200) per solve, against the separate launches: N = 4002, five steps: 182 us (409); N = 1002, three to
// four steps: 38 us (about 105, with the gaps).
// In a batch a team of CTAs takes one block after another, so that no stage waits for the slowest block between
// its products: four stages of 24 blocks of 362 to 1442 unknowns 5.16 -> 4.16 ms, of 256 of them 53.1 -> 51.0 ms
// (the matrices then come from HBM either way: 31 B per clock and SM; of one stage of 24 blocks 386 of the 514 MB that
// its products read).
#include <math.h>

#include <algorithm>
#include <vector>

#include "ctx.h"
#include "resident.cuh"

namespace bemb {

namespace {

constexpr int RF_D = 16;        // copies in flight per thread (131 KB per SM), in groups of RF_U columns
constexpr int RF_U = 4;
constexpr double BR_FIXED = 4.6e4;  // batch: a block's start and exchanges, in matrix elements of one CTA

// One system and this CTA's place in it.
struct RSys {
    int n, ldg, ldx, rows, row0;
    const double* A;
    const float* X;
    const double* b;
    const double* r;         // b - G x for the given x, or null
    double* x;               // start value, solution
    ulonglong2* ex;          // exchange slots of one parity
    long long ex_other;      // distance to those of the other
    unsigned long long seq;  // sequence numbers start above this
};
struct RRule {
    int kmax;
    double tol, strict, slow;  // stop at strict tol, or one step past tol; or when a step above 1000 tol
    long long wait_limit;      // contracts by no more than slow
    float keep_g, keep_x;      // shares of G and X to keep in L2
};

// The refinement of one system by the CTAs that share it.  record(step, rel, last) is called by every thread
// with each relative residual; *steps receives the corrections made.  False when an exchange wait ran out: x
// then stays as it was in this CTA's rows.
template <int K, typename Record>
__device__ bool refine_system(const RSys& a, const RRule& q, double* smem, int nv, int npart, double* bb_out,
                              int* steps, const Record& record) {
    const int n = a.n, tid = threadIdx.x, rows = a.rows, lane = tid & 31;
    const int row0 = a.row0, nr = max(0, min(rows, n - row0));
    double2* ring = reinterpret_cast<double2*>(smem) + tid;  // slot d at d RB_T
    double *vec = smem + (size_t)2 * RF_D * RB_T, *part = vec + nv, *red = part + npart;
    // G: two rows per copy; X: four
    const int pg = rows / 2, cg = RB_T / pg, ig = tid % pg * 2, jg = tid / pg, nkg = (n + RF_U * cg - 1) / (RF_U * cg);
    const int px = rows / 4, cx = RB_T / px, ix = tid % px * 4, jx = tid / px, nkx = (n + RF_U * cx - 1) / (RF_U * cx);
    const bool ong = jg < cg && ig < nr, onx = jx < cx && ix < nr;
    uint64_t polg, polx;
    asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, %1;" : "=l"(polg) : "f"(q.keep_g));
    asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, %1;" : "=l"(polx) : "f"(q.keep_x));
    // the stream: products with G and X in turn, columns jg + k cg and jx + k cx, RF_U at a time
    const double* gsrc = a.A + (size_t)min(jg, n - 1) * a.ldg + (ong ? row0 + ig : 0);
    const float* xsrc = a.X + (size_t)min(jx, n - 1) * a.ldx + (onx ? row0 + ix : 0);
    bool nextx = a.r != nullptr;
    int k_next = 0, slot = 0;
    auto advance = [&](int d) {
#pragma unroll
        for (int u = 0; u < RF_U; ++u) {
            const int k = k_next * RF_U + u;
            if (nextx) {
                if (onx)
                    ring_copy(ring + (d + u) * RB_T, reinterpret_cast<const double*>(xsrc + (size_t)k * cx * a.ldx),
                              jx + k * cx < n, polx);
            } else if (ong) {
                ring_copy(ring + (d + u) * RB_T, gsrc + (size_t)k * cg * a.ldg, jg + k * cg < n, polg);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++k_next == (nextx ? nkx : nkg)) {
            k_next = 0;
            nextx = !nextx;
        }
    };
#pragma unroll
    for (int d = 0; d < RF_D; d += RF_U) advance(d);
    for (int e = n + tid; e < nv; e += RB_T) vec[e] = 0.0;  // read with the zero columns past n
    double x[K], r[K];
    double bb = 0.0, rr = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int e = tid + k * RB_T;
        x[k] = r[k] = 0.0;
        if (e < n) {
            const double be = __ldg(a.b + e);
            bb += be * be;
            x[k] = __ldcg(a.x + e);
            if (a.r) r[k] = __ldg(a.r + e);
            rr += r[k] * r[k];
        }
    }
    cta_sums(red, bb, rr, true, bb, rr);
    unsigned long long seq = a.seq;
    double rel = sqrt(rr / bb), last = 0.0;
    int step = 0;
    bool ok = true, xturn = a.r != nullptr, reached = false;
    if (bb != 0.0)
        for (;;) {
            if (xturn) {  // a residual is at hand: converged, stuck or out of steps, or one more correction
                record(step, rel, last);
                if (rel <= q.strict * q.tol || reached || step == q.kmax ||
                    (step > 0 && last > 1e3 * q.tol && !(rel < q.slow * last)))
                    break;
                reached = rel <= q.tol;
            }
            // the own rows of G x or X r
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (tid + k * RB_T < n) vec[tid + k * RB_T] = xturn ? r[k] : x[k];
            __syncthreads();
            const int cs = xturn ? cx : cg;
            if (xturn) {
                for (int k = 0; k < nkx; ++k) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(RF_D / RF_U - 1) : "memory");
                    const double* vc = vec + jx + k * RF_U * cx;
                    float4 v[RF_U];
                    double xv[RF_U];
#pragma unroll
                    for (int u = 0; u < RF_U; ++u) {
                        v[u] = *reinterpret_cast<const float4*>(ring + (slot + u) * RB_T);
                        xv[u] = vc[u * cx];
                    }
#pragma unroll
                    for (int u = 0; u < RF_U; ++u) {
                        acc[0] = fma((double)v[u].x, xv[u], acc[0]);
                        acc[1] = fma((double)v[u].y, xv[u], acc[1]);
                        acc[2] = fma((double)v[u].z, xv[u], acc[2]);
                        acc[3] = fma((double)v[u].w, xv[u], acc[3]);
                    }
                    advance(slot);
                    slot = slot + RF_U == RF_D ? 0 : slot + RF_U;
                }
                if (onx)
#pragma unroll
                    for (int h = 0; h < 4; ++h) part[(ix + h) * (cs + 1) + jx] = acc[h];
            } else {
                for (int k = 0; k < nkg; ++k) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(RF_D / RF_U - 1) : "memory");
                    const double* vc = vec + jg + k * RF_U * cg;
                    double2 v[RF_U];
                    double xv[RF_U];
#pragma unroll
                    for (int u = 0; u < RF_U; ++u) {
                        v[u] = ring[(slot + u) * RB_T];
                        xv[u] = vc[u * cg];
                    }
#pragma unroll
                    for (int u = 0; u < RF_U; ++u) {
                        acc[0] = fma(v[u].x, xv[u], acc[0]);
                        acc[1] = fma(v[u].y, xv[u], acc[1]);
                    }
                    advance(slot);
                    slot = slot + RF_U == RF_D ? 0 : slot + RF_U;
                }
                if (ong) {
                    part[ig * (cs + 1) + jg] = acc[0];
                    part[(ig + 1) * (cs + 1) + jg] = acc[1];
                }
            }
            __syncthreads();
            ++seq;
            ulonglong2* slots = a.ex + (seq & 1 ? a.ex_other : 0);
            for (int w = tid >> 5; w < nr; w += RB_WARPS) {
                double s = 0.0;
                for (int k = lane; k < cs; k += 32) s += part[w * (cs + 1) + k];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) slot_store(slots + row0 + w, s, seq);
            }
            double t[K];
            ok = collect<K>(slots, n, seq, q.wait_limit, t);
            if (xturn) {
#pragma unroll
                for (int k = 0; k < K; ++k) x[k] += t[k];
                ++step;
                if (__syncthreads_or(!ok)) {
                    ok = false;
                    break;
                }
            } else {
                double s = 0.0, dummy;
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (tid + k * RB_T < n) {
                        r[k] = __ldg(a.b + tid + k * RB_T) - t[k];
                        s += r[k] * r[k];
                    }
                if (!cta_sums(red, s, 0.0, ok, s, dummy)) {
                    ok = false;
                    break;
                }
                last = rel;
                rel = sqrt(s / bb);
            }
            xturn = !xturn;
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok) return false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int e = tid + k * RB_T;
        if (e >= row0 && e < row0 + nr) a.x[e] = bb != 0.0 ? x[k] : 0.0;
    }
    *bb_out = bb;
    *steps = step;
    return true;
}

// One system over all CTAs.  out: |b|^2, steps, the launch's number if a wait ran out, then |r_k| / |b|.
template <int K>
__global__ void __launch_bounds__(RB_T, 1)
    k_refine_resident(RSys a, const RRule q, int nv, int npart, double* out, double number) {
    extern __shared__ __align__(16) double smem[];
    a.row0 = blockIdx.x * a.rows;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    double bb;
    int steps;
    const auto record = [&](int step, double rel, double) {
        if (first) out[3 + step] = rel;
    };
    if (!refine_system<K>(a, q, smem, nv, npart, &bb, &steps, record)) {
        if (threadIdx.x == 0) out[2] = number;
    } else if (first) {
        out[0] = bb;
        out[1] = steps;
    }
}

struct BRArgs {
    const BlockInfo* blk;
    const int *list, *off;   // the teams' blocks: list[off[t]] ... list[off[t + 1] - 1]
    const long long* xoff;   // the blocks' inverses in Xpad, negative: in X at their matrix's place
    const double* A;
    const float *X, *Xpad;
    const double* b;
    double* x;
    ulonglong2* ex;
    long long nverts;
    const unsigned long long* number;  // of this launch
    double *st, *err;                  // BSTAT_W statistics per block; set when a wait ran out
    int* conv;
    int team, nv, npart;
};

// A batch: teams of CTAs take their blocks one after the other.  The steps after a block's first find in L2 what is
// left there of its G and X beside the other teams' blocks: a quarter of the reads with 24 blocks, next to nothing
// in a large sweep.
template <int K>
__global__ void __launch_bounds__(RB_T, 1) k_refine_batch(const BRArgs a, const RRule q) {
    extern __shared__ __align__(16) double smem[];
    const int t = blockIdx.x / a.team, rank = blockIdx.x % a.team;
    const bool first = rank == 0 && threadIdx.x == 0;
    const unsigned long long seq = *a.number << 32;
    for (int e = a.off[t]; e < a.off[t + 1]; ++e) {
        const int k = a.list[e];
        const BlockInfo B = a.blk[k];
        RSys s;
        s.n = s.ldg = B.n;
        s.ldx = (B.n + 3) & ~3;
        s.rows = ((B.n + a.team - 1) / a.team + 3) & ~3;
        s.row0 = rank * s.rows;
        s.A = a.A + B.mbase;
        const long long xo = a.xoff[k];
        s.X = xo < 0 ? a.X + B.mbase : a.Xpad + xo;
        s.b = a.b + B.vbase;
        s.r = nullptr;
        s.x = a.x + B.vbase;
        s.ex = a.ex + B.vbase;
        s.ex_other = a.nverts;
        s.seq = seq;
        double* st = a.st + (size_t)BSTAT_W * k;
        double rho = 0.0, bb;
        int steps;
        const auto record = [&](int step, double rel, double last) {
            if (step > 0 && last > 1e3 * q.tol) rho = fmax(rho, rel / last);
            if (!first) return;
            if (step == 0) st[BS_FIRST] = rel;
            st[BS_LAST] = rel;
            st[BS_RHO] = rho;
            st[BS_CONV] = rel <= q.tol ? 1.0 : 0.0;
        };
        if (first) st[BS_FIRST] = st[BS_LAST] = st[BS_RHO] = 0.0;
        if (!refine_system<K>(s, q, smem, a.nv, a.npart, &bb, &steps, record)) {
            if (threadIdx.x == 0) *a.err = 1.0;
            return;
        }
        if (first) {
            st[BS_BB] = bb;
            st[BS_STEPS] = steps;
            if (bb == 0.0) st[BS_CONV] = 1.0;
            a.conv[k] = st[BS_CONV] != 0.0;
        }
        __syncthreads();  // the shared memory is free for the next block
    }
}

__global__ void k_next_number(unsigned long long* number) { ++*number; }

template <typename F>
cudaError_t rr_coop(F kernel, std::atomic<uint64_t>& ready, void** args, int grid, size_t smem, cudaStream_t s) {
    if (!once_per_device(ready, [kernel] {
            return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RB_SMEM) == cudaSuccess;
        }))
        return cudaErrorUnknown;
    return cudaLaunchCooperativeKernel((void*)kernel, grid, RB_T, args, smem, s);
}
template <int K>
cudaError_t rr_launch(void** args, bool batch, int grid, size_t smem, cudaStream_t s) {
    static std::atomic<uint64_t> one{0}, many{0};
    return batch ? rr_coop(k_refine_batch<K>, many, args, grid, smem, s)
                 : rr_coop(k_refine_resident<K>, one, args, grid, smem, s);
}
cudaError_t rr_launch_n(int n, void** args, bool batch, int grid, size_t smem, cudaStream_t s) {
    const int K = (n + RB_T - 1) / RB_T;
    return K <= 1   ? rr_launch<1>(args, batch, grid, smem, s)
           : K <= 2 ? rr_launch<2>(args, batch, grid, smem, s)
           : K <= 4 ? rr_launch<4>(args, batch, grid, smem, s)
           : K <= 8 ? rr_launch<8>(args, batch, grid, smem, s)
                    : rr_launch<12>(args, batch, grid, smem, s);
}

// Shared memory of a system of n unknowns over CTAs of `rows` rows: nv, npart grow to its needs.
void rr_sizes(int n, int rows, int* nv, int* npart) {
    const int cg = RB_T / (rows / 2), cx = RB_T / (rows / 4);
    const int ug = RF_U * cg, ux = RF_U * cx;
    const int cols = std::max((n + ug - 1) / ug * ug, (n + ux - 1) / ux * ux);
    *nv = std::max(*nv, (cols + cx + 1) & ~1);  // idle threads read a little past their columns
    *npart = std::max(*npart, rows * (std::max(cg, cx) + 1));
}
size_t rr_smem(int nv, int npart) { return sizeof(double) * ((size_t)2 * RF_D * RB_T + nv + npart + 2 * RB_WARPS); }

}  // namespace

// X for the streams: columns on 16 bytes.  A copy with a padded stride unless n is a multiple of four.
int refine_resident_inverse(Ctx& c, cudaStream_t s) {
    const size_t n = (size_t)c.topo.N, ld = (n + 3) & ~(size_t)3;
    if (!c.Xpad) return BEM_OK;
    BEM_CUDA(c, cudaMemcpy2DAsync(c.Xpad, sizeof(float) * ld, c.Xinv, sizeof(float) * n, sizeof(float) * n, n,
                                  cudaMemcpyDeviceToDevice, s));
    return BEM_OK;
}
size_t refine_resident_words(int64_t n) { return n <= RB_MAX_N && n % 4 ? (size_t)n * ((n + 3) & ~(size_t)3) : 0; }

bool refine_resident_fits(const Ctx& c) {
    return c.rfres_ok && c.rbicg && c.LU && c.topo.N <= RB_MAX_N && (c.topo.N % 4 == 0 || c.Xpad);
}

// One launch over the system a (n, G, X and their strides, b, x, r set).
static int rr_round(Ctx& c, RSys& a, const RRule& q, double* out, unsigned long long* number, cudaStream_t s) {
    int sms = 0, coop = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device);
    if (!coop) return BEM_ERR_CUDA;
    // 16 rows as in bicg_resident.cu, more where the SMs run out; a multiple of eight, so that a CTA's part of a
    // column of X is whole sectors: 32 rows on 126 SMs at N = 4002 39.4 us per step with the first residual's
    // share, 28 rows on 143 SMs 41.0; N = 5292: 69.1 and 71.9; N = 4842: 63.9 and 63.0
    a.rows = std::max(16, ((a.n + sms - 1) / sms + 7) & ~7);
    const int grid = (a.n + a.rows - 1) / a.rows;
    int nv = 0, npart = 0;
    rr_sizes(a.n, a.rows, &nv, &npart);
    const size_t smem = rr_smem(nv, npart);
    if (smem > RB_SMEM) return BEM_ERR_CUDA;
    a.ex = reinterpret_cast<ulonglong2*>(c.rbicg);
    a.ex_other = a.n;
    *number = ++c.rbicg_solves;
    a.seq = *number << 32;
    double id = (double)*number;
    void* args[] = {&a, (void*)&q, &nv, &npart, &out, &id};
    KLAUNCH();
    if (rr_launch_n(a.n, args, false, grid, smem, s) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    return BEM_OK;
}

// A rule with the shares of G and X to keep in L2: RB_KEEP bytes, G first.  At N = 4002 with rows of 32, per step:
// 64 MB of G 33.7 us, 32 MB of G and of X 34.6, X alone 36.6, all of X and 32 MB of G 37.8.
static RRule rr_rule(const Ctx& c, int n, int kmax, double tol, double strict, double slow) {
    const double g = 8.0 * n * n, x = 4.0 * n * n;
    return {kmax, tol, strict, slow, c.wait_limit, (float)std::min(1.0, RB_KEEP / g),
            (float)std::max(0.0, std::min(1.0, (RB_KEEP - g) / x))};
}

// One round of at most kmax steps from x; out (3 + kmax + 1 doubles on the device, as k_refine_resident leaves
// them); *number: the launch's.  BEM_ERR_CUDA: the launch failed, nothing done.
int refine_resident(Ctx& c, const double* A, const double* b, double* x, const double* r, bool r_ready, int kmax,
                    double tol, double slow, double* out, unsigned long long* number, cudaStream_t s) {
    const int n = (int)c.topo.N;
    RSys a{};
    a.n = n;
    a.ldg = n;
    a.ldx = (n + 3) & ~3;
    a.X = c.Xpad ? c.Xpad : c.Xinv;
    if (n % 2 || reinterpret_cast<uintptr_t>(A) % 16) {  // copies of 16 bytes: a matrix with an even stride
        a.ldg = (n + 1) & ~1;
        BEM_CUDA(c, cudaMemcpy2DAsync(c.LU, sizeof(double) * a.ldg, A, sizeof(double) * n, sizeof(double) * n, n,
                                      cudaMemcpyDeviceToDevice, s));
        A = c.LU;
    }
    a.A = A;
    a.b = b;
    a.r = r_ready ? r : nullptr;
    a.x = x;
    // a tenth of the tolerance, or one step past it: the last step is cheap, and a solve that only just meets
    // the tolerance would leave the solution less exact than the rounds of separate launches do
    const RRule q = rr_rule(c, n, kmax, tol, tol >= 1e-13 ? 0.1 : 1.0, slow);
    return rr_round(c, a, q, out, number, s);
}

// blockIdx.z = 0: G^T into gt (stride ldg); 1: X^T into xt (stride ldx).
__global__ void __launch_bounds__(256)
    k_transpose_gx(int n, const double* __restrict__ G, const float* __restrict__ X, double* __restrict__ gt, int ldg,
                   float* __restrict__ xt, int ldx) {
    __shared__ double tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32, lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
    const bool g = blockIdx.z == 0;
    for (int k = ly; k < 32; k += 8)
        if (r0 + lx < n && c0 + k < n) {
            const size_t e = (size_t)(c0 + k) * n + r0 + lx;
            tile[k][lx] = g ? G[e] : (double)X[e];
        }
    __syncthreads();
    for (int k = ly; k < 32; k += 8)
        if (c0 + lx < n && r0 + k < n) {
            if (g)
                gt[(size_t)(r0 + k) * ldg + c0 + lx] = tile[lx][k];
            else
                xt[(size_t)(r0 + k) * ldx + c0 + lx] = (float)tile[lx][k];
        }
}

// The same round for G^T y = b through the transpose of the approximate inverse; xt: n columns of
// (n + 3) & ~3 floats.  renewed: G or the inverse changed, the transposes are made; first: y starts from zero.
int refine_resident_transposed(Ctx& c, const double* G, const double* b, double* y, bool renewed, bool first, float* xt,
                               int kmax, double tol, double* out, unsigned long long* number, cudaStream_t s) {
    const int n = (int)c.topo.N, nt = (n + 31) / 32;
    RSys a{};
    a.n = n;
    a.ldg = (n + 1) & ~1;
    a.ldx = (n + 3) & ~3;
    a.A = c.LU;
    a.X = xt;
    a.b = b;
    a.r = first ? b : nullptr;
    a.x = y;
    if (renewed) KLAUNCH(), k_transpose_gx<<<dim3(nt, nt, 2), 256, 0, s>>>(n, G, c.Xinv, c.LU, a.ldg, xt, a.ldx);
    if (first) BEM_CUDA(c, cudaMemsetAsync(y, 0, sizeof(double) * n, s));
    // the separate launches always run six steps: two orders below the tolerance, or one step past it
    const RRule q = rr_rule(c, n, kmax, tol, tol >= 1e-13 ? 0.01 : 1.0, INFINITY);
    return rr_round(c, a, q, out, number, s);
}

// The batch's plan: teams of CTAs and their blocks (longest first, each to the team with the least work), the
// padded inverses' places.  Every block even-sized (G's copies of 16 bytes) and within RB_MAX_N, or no plan.
int refine_batch_setup(Ctx& c) {
    c.bteam = 0;
    int sms = 0, coop = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device);
    long long xtot = 0;
    std::vector<long long> xoff;
    for (const BlockInfo& B : c.h_blk) {
        if (B.n % 2 || B.n > RB_MAX_N) return BEM_OK;
        xoff.push_back(B.n % 4 ? xtot : -1);
        if (B.n % 4) xtot += (long long)B.n * ((B.n + 3) & ~3);
    }
    std::vector<int> order((size_t)c.nblk);
    for (int b = 0; b < c.nblk; ++b) order[(size_t)b] = b;
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return c.h_blk[(size_t)a].n > c.h_blk[(size_t)b].n; });
    // The team size whose longest list of blocks is shortest, the largest blocks first to the least loaded team.
    // Small teams waste less on exchanges, large ones leave less of the chip idle behind the last block.  Four
    // stages by team size, ms: 24 blocks of 362 to 1442 unknowns: 4: 5.98, 8: 4.51, 12: 4.16, 16: 4.21, 24: 4.37;
    // 256 of the same: 51.2, 50.9, 52.1, 52.1, 53.8; 64 of 162 to 642: 3.71, 3.96, 4.23, 4.57, 5.20; three:
    // 11.7, 6.3, 5.3, 4.5, 3.9 and 49: 3.36.
    int team = 0, teams = 0;
    std::vector<std::vector<int>> mine;
    double best = INFINITY;
    std::vector<int> sizes{4, 6, 8, 12, 16, 24};
    if (sms / c.nblk > 24) sizes.push_back(sms / c.nblk);
    for (int t : sizes) {
        const int nt = sms / t;
        int nv = 0, npart = 0;
        if ((c.bmax_n + t - 1) / t > 2 * RB_T - 4) continue;  // two rows of G per thread at most
        for (const BlockInfo& B : c.h_blk) rr_sizes(B.n, ((B.n + t - 1) / t + 3) & ~3, &nv, &npart);
        if (!coop || nt < 1 || rr_smem(nv, npart) > RB_SMEM) continue;
        std::vector<std::vector<int>> lists((size_t)nt);
        std::vector<double> load((size_t)nt, 0.0);
        for (int b : order) {
            const size_t k = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
            lists[k].push_back(b);
            const double n = c.h_blk[(size_t)b].n;
            load[k] += n * n / t + BR_FIXED;
        }
        const double longest = *std::max_element(load.begin(), load.end());
        if (longest < best) {
            best = longest;
            team = t;
            teams = nt;
            mine = lists;
            c.bnv = nv;
            c.bnpart = npart;
        }
    }
    if (!team) return BEM_OK;
    std::vector<int> list, off{0};
    for (const auto& m : mine) {
        list.insert(list.end(), m.begin(), m.end());
        off.push_back((int)list.size());
    }
    int rc;
    if ((rc = upload_vec(c, &c.blist, list)) || (rc = upload_vec(c, &c.boff, off)) ||
        (rc = upload_vec(c, &c.bxoff, xoff)) ||
        (rc = dalloc(c, &c.bslots, 4 * (size_t)c.h_blk.back().vbase + 4 * (size_t)c.h_blk.back().n)) ||
        (rc = dalloc(c, &c.bnumber, 1)) || (rc = dalloc(c, &c.Xbpad, (size_t)xtot))) {
        if (rc != BEM_ERR_NOMEM) return rc;
        cudaGetLastError();  // no memory for the copies: the separate launches
        return BEM_OK;
    }
    c.h_bxoff = xoff;
    BEM_CUDA(c, cudaMemset(c.bslots, 0, sizeof(double) * 4 * (size_t)(c.h_blk.back().vbase + c.h_blk.back().n)));
    BEM_CUDA(c, cudaMemset(c.bnumber, 0, sizeof(unsigned long long)));
    c.bteam = team;
    c.bteams = teams;
    return BEM_OK;
}

// After every change of block b's inverse.
int refine_batch_inverse(Ctx& c, int b, cudaStream_t s) {
    if (!c.bteam || c.h_bxoff[(size_t)b] < 0) return BEM_OK;
    const BlockInfo& B = c.h_blk[(size_t)b];
    const size_t n = (size_t)B.n, ld = (n + 3) & ~(size_t)3;
    BEM_CUDA(c, cudaMemcpy2DAsync(c.Xbpad + c.h_bxoff[(size_t)b], sizeof(float) * ld, c.Xb + B.mbase, sizeof(float) * n,
                                  sizeof(float) * n, n, cudaMemcpyDeviceToDevice, s));
    return BEM_OK;
}

// The batched solve; BEM_ERR_CUDA: the launch failed, nothing done.  Expired waits: *err on the device.
int refine_batch(Ctx& c, const double* A, const double* b, double* x, int kmax, double tol, double* err, cudaStream_t s) {
    BRArgs a{c.blk, c.blist, c.boff, c.bxoff, A, c.Xb, c.Xbpad, b, x, reinterpret_cast<ulonglong2*>(c.bslots),
             (long long)c.topo.N, c.bnumber, c.bstat, err, c.bconv, c.bteam, c.bnv, c.bnpart};
    // Everything marked to stay is no preference, and none helps: a share for G changed nothing
    RRule q{kmax, tol, 1.0, INFINITY, c.wait_limit, 1.0f, 1.0f};
    KLAUNCH(), k_next_number<<<1, 1, 0, s>>>(c.bnumber);
    void* args[] = {&a, &q};
    KLAUNCH();
    if (rr_launch_n(c.bmax_n, args, true, c.bteam * c.bteams, rr_smem(c.bnv, c.bnpart), s) != cudaSuccess) {
        cudaGetLastError();
        return BEM_ERR_CUDA;
    }
    return BEM_OK;
}

}  // namespace bemb
