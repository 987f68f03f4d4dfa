// BIE operator, right-hand side, restarted GMRES, polarization energy and the whole solve.
//
//   bie_matvec     dmapping (electric.cpp:294-388): densities -> fused FMM -> combine
//   k_rhs          load (electric.cpp:395-412), direct atom sums (k_rhs32: FP32, mixed path)
//   gmres          GMRES (gmres.cpp:50-164): modified Gram-Schmidt Arnoldi on the device with
//                  fixed-order (deterministic) reductions; Givens rotations and the small
//                  triangular solve on the host in FP64, as in the reference
//   polarize       polarizeMap + energy (electric.cpp:442-505)
//   solve          main.cpp:45-77 for an explicit geometry
// Mixed precision (IBIM_PRECISION_MIXED): the same GMRES runs on the FP32 operator inside an
// FP64 iterative-refinement loop whose residual uses the FP64 operator (IBIM_PRECISION_FP64_TC:
// FP64 near field and X list, V-list M2L as exact BF16 digit products on the tensor cores).

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>

#include "fmm_common.cuh"
#include "solve.cuh"

namespace ibim {

namespace {

constexpr int RED_BLOCKS = 512;  // fixed reduction width: results independent of the GPU size
constexpr int RED_THREADS = 256;

// m_a = x n_a w, psi = x' w (electric.cpp:324-329), tree order.
__global__ void k_densities(long n, const double *__restrict__ x, const double *__restrict__ nx,
                            const double *__restrict__ ny, const double *__restrict__ nz,
                            const double *__restrict__ w, double *dens) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double xi = x[i], wi = w[i];
        dens[i] = xi * nx[i] * wi;
        dens[n + i] = xi * ny[i] * wi;
        dens[2 * n + i] = xi * nz[i] * wi;
        dens[3 * n + i] = x[n + i] * wi;
    }
}

// out1 = phi + F / (1/2 (1 + eE/eI)); out2 = dphi + n.G / (1/2 (1 + eI/eE)) (electric.cpp:369-384).
__global__ void k_combine(long n, const double *__restrict__ x, const double *__restrict__ f,
                          const double *__restrict__ nx, const double *__restrict__ ny, const double *__restrict__ nz,
                          double e1, double e2, double *y) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double ng = nx[i] * f[n + i] + ny[i] * f[2 * n + i] + nz[i] * f[3 * n + i];
        y[i] = x[i] + f[i] / e1;
        y[n + i] = x[n + i] + ng / e2;
    }
}

// Right-hand side (electric.cpp:395-412) at tree-ordered tube points; atoms staged in shared memory.
__global__ void __launch_bounds__(256) k_rhs(long n, const double *__restrict__ px, const double *__restrict__ py,
                                             const double *__restrict__ pz, const double *__restrict__ nx,
                                             const double *__restrict__ ny, const double *__restrict__ nz,
                                             const double *__restrict__ atoms, int natoms, double c1, double c2,
                                             double *b) {
    __shared__ double A[4][256];
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    double X = 0, Y = 0, Z = 0, NX = 0, NY = 0, NZ = 0;
    if (i < n) { X = px[i]; Y = py[i]; Z = pz[i]; NX = nx[i]; NY = ny[i]; NZ = nz[i]; }
    double b1 = 0., b2 = 0.;
    for (int a0 = 0; a0 < natoms; a0 += 256) {
        const int cnt = min(256, natoms - a0);
        __syncthreads();
        if (threadIdx.x < cnt)
            for (int q = 0; q < 4; ++q) A[q][threadIdx.x] = atoms[4 * (a0 + threadIdx.x) + q];
        __syncthreads();
        if (i < n)
            for (int a = 0; a < cnt; ++a) {
                const double dx = X - A[0][a], dy = Y - A[1][a], dz = Z - A[2][a];
                const double d = dx * dx + dy * dy + dz * dz;
                const double ir = rsqrt64(d);  // 1 / r (electric.cpp:401-409 divides by r and r^3)
                b1 += A[3][a] * c1 * ir;
                b2 -= A[3][a] * c2 * (ir * ir * ir) * (NX * dx + NY * dy + NZ * dz);
            }
    }
    if (i < n) {
        b[i] = b1;
        b[n + i] = b2;
    }
}

// load in FP32 for the mixed path: coordinates relative to the block's first point (differences
// taken in FP64, so each point-atom offset carries FP32 rounding only), rsqrt in FP32, per-tile
// partial sums added with Kahan compensation; the result is stored in FP64.
__global__ void __launch_bounds__(256) k_rhs32(long n, const double *__restrict__ px, const double *__restrict__ py,
                                               const double *__restrict__ pz, const double *__restrict__ nx,
                                               const double *__restrict__ ny, const double *__restrict__ nz,
                                               const double *__restrict__ atoms, int natoms, double c1, double c2,
                                               double *b) {
    __shared__ float A[4][256];
    __shared__ double org[3];
    const long i0 = blockIdx.x * (long)blockDim.x;
    const long i = i0 + threadIdx.x;
    if (threadIdx.x == 0) {
        org[0] = px[i0];
        org[1] = py[i0];
        org[2] = pz[i0];
    }
    __syncthreads();
    float X = 0.f, Y = 0.f, Z = 0.f, NX = 0.f, NY = 0.f, NZ = 0.f;
    if (i < n) {
        X = (float)(px[i] - org[0]);
        Y = (float)(py[i] - org[1]);
        Z = (float)(pz[i] - org[2]);
        NX = (float)nx[i];
        NY = (float)ny[i];
        NZ = (float)nz[i];
    }
    float s1 = 0.f, k1 = 0.f, s2 = 0.f, k2 = 0.f;
    for (int a0 = 0; a0 < natoms; a0 += 256) {
        const int cnt = min(256, natoms - a0);
        __syncthreads();
        if (threadIdx.x < cnt) {
            const double *at = atoms + 4 * (long)(a0 + threadIdx.x);
            A[0][threadIdx.x] = (float)(at[0] - org[0]);
            A[1][threadIdx.x] = (float)(at[1] - org[1]);
            A[2][threadIdx.x] = (float)(at[2] - org[2]);
            A[3][threadIdx.x] = (float)at[3];
        }
        __syncthreads();
        if (i < n) {
            float p1 = 0.f, p2 = 0.f;
            for (int a = 0; a < cnt; ++a) {
                const float dx = X - A[0][a], dy = Y - A[1][a], dz = Z - A[2][a];
                const float ir = rsqrtf(dx * dx + dy * dy + dz * dz);
                const float qi = A[3][a] * ir;
                p1 += qi;
                p2 += qi * ir * ir * (NX * dx + NY * dy + NZ * dz);
            }
            float y = p1 - k1, t = s1 + y;
            k1 = (t - s1) - y;
            s1 = t;
            y = p2 - k2;
            t = s2 + y;
            k2 = (t - s2) - y;
            s2 = t;
        }
    }
    if (i < n) {
        b[i] = c1 * (double)(s1 - k1);
        b[n + i] = -c2 * (double)(s2 - k2);
    }
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double sh[RED_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.;
    if (threadIdx.x == 0)
        for (int w = 0; w < RED_THREADS / 32; ++w) s += sh[w];
    __syncthreads();
    return s;  // valid in thread 0
}

// Reduce RED_BLOCKS partials in a fixed order; every block computes the same value.
__device__ __forceinline__ double reduce_partials(const double *__restrict__ part) {
    __shared__ double v;
    double s = 0.;
    for (int q = threadIdx.x; q < RED_BLOCKS; q += RED_THREADS) s += part[q];
    s = block_sum(s);
    if (threadIdx.x == 0) v = s;
    __syncthreads();
    return v;
}

__global__ void __launch_bounds__(RED_THREADS) k_dot(long n, const double *__restrict__ a, const double *__restrict__ b,
                                                     double *part) {
    double s = 0.;
    for (long i = blockIdx.x * (long)RED_THREADS + threadIdx.x; i < n; i += (long)RED_BLOCKS * RED_THREADS)
        s += a[i] * b[i];
    s = block_sum(s);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// MGS step: h = <w, v_prev> (from the partials), w -= h v_prev, then partial <w, v_next>
// (or <w, w> when v_next is null).  h is stored in hcol[slot].
__global__ void __launch_bounds__(RED_THREADS) k_mgs(long n, const double *__restrict__ part_in, double *w,
                                                     const double *__restrict__ v_prev,
                                                     const double *__restrict__ v_next, double *part_out,
                                                     double *hcol, int slot) {
    const double h = reduce_partials(part_in);
    if (blockIdx.x == 0 && threadIdx.x == 0) hcol[slot] = h;
    double s = 0.;
    for (long i = blockIdx.x * (long)RED_THREADS + threadIdx.x; i < n; i += (long)RED_BLOCKS * RED_THREADS) {
        const double wi = w[i] - h * v_prev[i];
        w[i] = wi;
        s += wi * (v_next ? v_next[i] : wi);
    }
    s = block_sum(s);
    if (threadIdx.x == 0) part_out[blockIdx.x] = s;
}

// v = w / ||w|| with ||w|| from the partials of <w, w>; ||w|| stored in hcol[slot].
__global__ void __launch_bounds__(RED_THREADS) k_normalize(long n, const double *__restrict__ part_in,
                                                           const double *__restrict__ w, double *v, double *hcol,
                                                           int slot) {
    const double nr = sqrt(reduce_partials(part_in));
    if (blockIdx.x == 0 && threadIdx.x == 0) hcol[slot] = nr;
    const double s = 1.0 / nr;
    for (long i = blockIdx.x * (long)RED_THREADS + threadIdx.x; i < n; i += (long)RED_BLOCKS * RED_THREADS)
        v[i] = w[i] * s;
}

// One Arnoldi step after w = A v_i in one launch: the modified Gram-Schmidt chain of k_dot, i + 1 times
// k_mgs and k_normalize, with the same sums in the same order.  The chain is serial (each coefficient
// needs the vector the last one left), so as i + 3 launches it cost their latency and three passes over
// w; here the blocks are resident together (a cooperative launch), keep their part of w in
// registers (R values a thread) and meet at a barrier between steps, which each costs one pass over v_k.
// A block is four of the separate launches' blocks ("lanes" of RED_THREADS threads), so that 128
// blocks at most, and for short vectors as few as hold values, take part in the barrier.
// 14 steps on 15 k points (n = 30 k): 1.43 -> 0.93 ms, 26 on 419 k: 5.8 -> 4.0 ms (with 512 blocks of 256 threads at
// the barrier: 1.06 and 4.3).
// bar[0] counts arrivals (base: before this launch); a wait that runs out sets bar[1] and goes on.
constexpr int ARN_LANES = 4, ARN_THREADS = ARN_LANES * RED_THREADS;
template <int R>
__global__ void __launch_bounds__(ARN_THREADS, 1) k_arnoldi(long n, int i, const double *__restrict__ w, double *V,
                                                            double *part, double *hcol, unsigned *bar, unsigned base) {
    __shared__ double sh[ARN_LANES][RED_THREADS / 32], total;
    const int g = threadIdx.x / RED_THREADS, l = threadIdx.x % RED_THREADS;
    const int blk = blockIdx.x * ARN_LANES + g, nblk = gridDim.x * ARN_LANES;  // of the separate launches
    const long t = blk * (long)RED_THREADS + l;
    constexpr long STRIDE = (long)RED_BLOCKS * RED_THREADS;
    double x[R];
    unsigned target = base;
    // block_sum's order within a lane; valid in its first thread
    auto lane_sum = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((l & 31) == 0) sh[g][l >> 5] = v;
        __syncthreads();
        double s = 0.;
        if (l == 0)
            for (int q = 0; q < RED_THREADS / 32; ++q) s += sh[g][q];
        return s;
    };
    // the lanes' partials of step k out, every block's in
    auto exchange = [&](double v, int k) {
        double *p = part + (k & 1) * RED_BLOCKS;
        const double s = lane_sum(v);
        if (l == 0) p[blk] = s;
        __syncthreads();
        target += gridDim.x;
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(bar, 1u);
            int left = 1 << 22;
            while ((int)(*(volatile unsigned *)bar - target) < 0 && --left > 0) {}
            if (left <= 0) bar[1] = 1u;
            __threadfence();
        }
        __syncthreads();
        double a = 0.;  // reduce_partials' order; the blocks that hold no values would add zeros
        if (g == 0)
            for (int q = l; q < nblk; q += RED_THREADS) a += __ldcg(p + q);
        a = lane_sum(a);
        if (threadIdx.x == 0) total = a;
        __syncthreads();
        return total;
    };
    double s = 0.;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const long e = t + q * STRIDE;
        x[q] = e < n ? w[e] : 0.;
        if (e < n) s += x[q] * V[e];
    }
    for (int k = 0; k <= i; ++k) {
        const double h = exchange(s, k);
        if (t == 0) hcol[k] = h;
        const double *vk = V + (long)k * n, *vn = vk + n;
        s = 0.;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const long e = t + q * STRIDE;
            if (e < n) {
                x[q] -= h * vk[e];
                s += x[q] * (k < i ? vn[e] : x[q]);
            }
        }
    }
    const double nr = sqrt(exchange(s, i + 1));
    if (t == 0) hcol[i + 1] = nr;
    const double f = 1.0 / nr;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const long e = t + q * STRIDE;
        if (e < n) V[(long)(i + 1) * n + e] = x[q] * f;
    }
}

const void *arnoldi_kernel(int R) {
    return R == 2 ? (const void *)k_arnoldi<2> : (R == 8 ? (const void *)k_arnoldi<8> : (const void *)k_arnoldi<16>);
}

// The registers a thread that hold vectors of length n, or 0 where the launches stay apart: vectors
// beyond 16 values a thread, or a device that cannot hold the blocks at once.
int arnoldi_regs(Ctx *c, long n) {
    const long per = div_up(n, (long)RED_BLOCKS * RED_THREADS);
    const int R = per <= 2 ? 2 : (per <= 8 ? 8 : (per <= 16 ? 16 : 0));
    if (R == 0) return 0;
    int b = 0;
    IBIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, arnoldi_kernel(R), ARN_THREADS, 0));
    return (long)b * c->num_sms >= RED_BLOCKS / ARN_LANES ? R : 0;
}

// x += sum_j y_j v_j (gmres.cpp:19-20, one daxpy per j in order).
__global__ void k_update(long n, int k, const double *__restrict__ y, const double *__restrict__ V, double *x) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        double s = x[i];
        for (int j = 0; j < k; ++j) s += y[j] * V[(long)j * n + i];
        x[i] = s;
    }
}

__global__ void k_sub(long n, const double *__restrict__ a, const double *__restrict__ b, double *c) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) c[i] = a[i] - b[i];
}

__global__ void k_axpy(long n, double a, const double *__restrict__ x, double *y) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) y[i] += a * x[i];
}

__global__ void k_permute(long n, const int *__restrict__ perm, const double *__restrict__ in, double *out, int scatter) {
    // scatter: out[perm[i]] = in[i]; gather: out[i] = in[perm[i]]
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        if (scatter)
            out[perm[i]] = in[i];
        else
            out[i] = in[perm[i]];
    }
}

inline int ew_grid(Ctx *c, long n) { return (int)std::max<long>(1, std::min<long>(8L * c->num_sms, div_up(n, 256))); }

}  // namespace

void permute(Ctx *c, long n, const int *perm, const double *in, double *out, bool scatter) {
    if (n <= 0) return;
    (count_launch(), k_permute<<<ew_grid(c, n), 256, 0, c->stream>>>(n, perm, in, out, scatter ? 1 : 0));
    IBIM_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------------------
// BIE operator
// ---------------------------------------------------------------------------------------

namespace {

bool matvec_graphs() {
    static const bool on = [] {
        const char *v = std::getenv("IBIM_GRAPHS");
        return !(v && v[0] == '0');
    }();
    return on;
}

void matvec_body(Plan &P, const ibim_kernel_params &kp, const double *x, double *y, int precision);

// The mixed matvec (25 of a solve's 26 products) as one CUDA graph: the first call with given
// kernel parameters runs the launches directly (it makes the plan's lazy set-up: operator images,
// near lists, workspaces), the second captures them on the context stream (the near field's fork
// to the second stream and its join are captured as dependencies) and every call from then on
// stages its input into gx, replays the graph and copies gy out.  Not while per-kernel profiling
// records events.  A capture that fails leaves the plan on direct launches.
bool matvec_graph(Plan &P, const ibim_kernel_params &kp, const double *x, double *y) {
    Ctx *c = P.ctx;
    if (!matvec_graphs() || c->prof_mask != 0 || P.mvg.failed) return false;
    Plan::MatvecGraph &G = P.mvg;
    const double key[5] = {kp.kappa, kp.dE, kp.dI, kp.tau, (double)kp.k3_scaled};
    if (std::memcmp(key, G.key, sizeof key) != 0) {
        if (G.exec) cudaGraphExecDestroy(G.exec);
        G.exec = nullptr;
        G.calls = 0;
        std::memcpy(G.key, key, sizeof key);
    }
    if (!G.exec && G.calls++ == 0) return false;
    const long n2 = 2 * P.ns;
    cudaStream_t s = c->stream;
    if (!G.exec) {
        if (!P.gx.ptr) {
            P.gx.alloc(n2, s);
            P.gy.alloc(n2, s);
        }
        IBIM_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        const long before = launch_count();
        cudaGraph_t g = nullptr;
        try {
            matvec_body(P, kp, P.gx.ptr, P.gy.ptr, IBIM_PRECISION_MIXED);
        } catch (...) {
            cudaStreamEndCapture(s, &g);
            if (g) cudaGraphDestroy(g);
            (void)cudaGetLastError();
            G.failed = true;
            return false;
        }
        const cudaError_t e = cudaStreamEndCapture(s, &g);
        count_launches(-(launch_count() - before));  // captured, not launched
        if (e != cudaSuccess || !g) {
            (void)cudaGetLastError();
            G.failed = true;
            return false;
        }
        size_t nn = 0;
        IBIM_CUDA(cudaGraphGetNodes(g, nullptr, &nn));
        std::vector<cudaGraphNode_t> nodes(nn);
        IBIM_CUDA(cudaGraphGetNodes(g, nodes.data(), &nn));
        G.kernels = 0;
        for (cudaGraphNode_t nd : nodes) {
            cudaGraphNodeType t;
            IBIM_CUDA(cudaGraphNodeGetType(nd, &t));
            G.kernels += t == cudaGraphNodeTypeKernel;
        }
        const cudaError_t ei = cudaGraphInstantiate(&G.exec, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) {
            (void)cudaGetLastError();
            G.exec = nullptr;
            G.failed = true;
            return false;
        }
        trace_mark("matvec graph captured");
    }
    IBIM_CUDA(cudaMemcpyAsync(P.gx.ptr, x, sizeof(double) * n2, cudaMemcpyDeviceToDevice, s));
    IBIM_CUDA(cudaGraphLaunch(G.exec, s));
    IBIM_CUDA(cudaMemcpyAsync(y, P.gy.ptr, sizeof(double) * n2, cudaMemcpyDeviceToDevice, s));
    count_launches(G.kernels);
    return true;
}

}  // namespace

void bie_matvec(Plan &P, const ibim_kernel_params &kp, const double *x, double *y, int precision) {
    IBIM_REQUIRE(!P.targets.empty() && P.targets[0]->self, "BIE operator needs a plan over the tube points");
    if (precision == IBIM_PRECISION_MIXED && matvec_graph(P, kp, x, y)) return;
    matvec_body(P, kp, x, y, precision);
}

namespace {

void matvec_body(Plan &P, const ibim_kernel_params &kp, const double *x, double *y, int precision) {
    Ctx *c = P.ctx;
    const long n = P.ns;
    (count_launch(), k_densities<<<ew_grid(c, n), 256, 0, c->stream>>>(n, x, P.snx.ptr, P.sny.ptr, P.snz.ptr, P.sw.ptr, P.dens4.ptr));
    IBIM_CHECK_LAUNCH();
    TargetSet &S = *P.targets[0];
    fmm_run(P, 0, kp, P.dens4.ptr, S.out4.ptr, precision);
    const double e1 = 0.5 * (1 + kp.dE / kp.dI), e2 = 0.5 * (1 + kp.dI / kp.dE);
    (count_launch(), k_combine<<<ew_grid(c, n), 256, 0, c->stream>>>(n, x, S.out4.ptr, P.snx.ptr, P.sny.ptr, P.snz.ptr, e1, e2, y));
    IBIM_CHECK_LAUNCH();
}

}  // namespace

void bie_densities(Plan &P, const double *x, double *dens4) {
    const long n = P.ns;
    (count_launch(), k_densities<<<ew_grid(P.ctx, n), 256, 0, P.ctx->stream>>>(n, x, P.snx.ptr, P.sny.ptr, P.snz.ptr,
                                                                               P.sw.ptr, dens4));
    IBIM_CHECK_LAUNCH();
}

static void rhs_launch(Ctx *c, long n, const double *x, const double *y, const double *z, const double *nx,
                       const double *ny, const double *nz, const ibim_kernel_params &kp, const double *atoms4_dev,
                       int natoms, double *b, cudaStream_t st, bool fp32) {
    const double e1 = 0.5 * (1 + kp.dE / kp.dI), e2 = 0.5 * (1 + kp.dI / kp.dE);
    const double c1 = 1.0 / (kp.dI * 4.0 * M_PI * e1), c2 = 1.0 / (kp.dI * 4.0 * M_PI * e2);
    ProfScope ps_(PROF_RHS, 20.0 * n * (double)natoms, 0., st);
    if (fp32)
        (count_launch(), k_rhs32<<<div_up(n, 256), 256, 0, st>>>(n, x, y, z, nx, ny, nz, atoms4_dev, natoms, c1, c2, b));
    else
        (count_launch(), k_rhs<<<div_up(n, 256), 256, 0, st>>>(n, x, y, z, nx, ny, nz, atoms4_dev, natoms, c1, c2, b));
    IBIM_CHECK_LAUNCH();
}

void bie_rhs(Plan &P, const ibim_kernel_params &kp, const double *atoms4_dev, int natoms, double *b) {
    rhs_launch(P.ctx, P.ns, P.sx.ptr, P.sy.ptr, P.sz.ptr, P.snx.ptr, P.sny.ptr, P.snz.ptr, kp, atoms4_dev, natoms, b,
               P.ctx->stream, P.precision == IBIM_PRECISION_MIXED);
}

void bie_rhs_tube(const Tube &t, const ibim_kernel_params &kp, const double *atoms4_dev, int natoms, double *b,
                  cudaStream_t st, int precision) {
    rhs_launch(t.ctx, t.n, t.x.ptr, t.y.ptr, t.z.ptr, t.nx.ptr, t.ny.ptr, t.nz.ptr, kp, atoms4_dev, natoms, b, st,
               precision == IBIM_PRECISION_MIXED);
}

// ---------------------------------------------------------------------------------------
// GMRES
// ---------------------------------------------------------------------------------------

namespace {

// gmres.cpp:23-43
void gen_rot(double dx, double dy, double &cs, double &sn) {
    if (dy == 0.0) {
        cs = 1.0;
        sn = 0.0;
    } else if (std::fabs(dy) > std::fabs(dx)) {
        const double t = dx / dy;
        sn = 1.0 / std::sqrt(1.0 + t * t);
        cs = t * sn;
    } else {
        const double t = dy / dx;
        cs = 1.0 / std::sqrt(1.0 + t * t);
        sn = t * cs;
    }
}
void apply_rot(double &dx, double &dy, double cs, double sn) {
    const double t = cs * dx + sn * dy;
    dy = -sn * dx + cs * dy;
    dx = t;
}

}  // namespace

Krylov::Krylov(Ctx *c, long n_, int m_) : ctx(c), n(n_), m(m_) {
    // between the matvecs, without a change of the SMs' split of L1 and shared memory
    static std::atomic<uint64_t> split;
    side_by_side(split, {(const void *)k_densities, (const void *)k_combine, (const void *)k_dot, (const void *)k_mgs,
                         (const void *)k_normalize, (const void *)k_update, (const void *)k_sub, (const void *)k_axpy,
                         (const void *)k_permute, (const void *)k_arnoldi<2>, (const void *)k_arnoldi<8>,
                         (const void *)k_arnoldi<16>});
    bar.alloc(2, c->stream);
    bar.zero();
    cudaStream_t s = c->stream;
    V.alloc((size_t)(m + 1) * n, s);
    w.alloc(n, s);
    r.alloc(n, s);
    part.alloc(2 * RED_BLOCKS, s);
    hcol.alloc(m + 2, s);
    ydev.alloc(m + 1, s);
    IBIM_CUDA(cudaMallocHost((void **)&hpin, sizeof(double) * (2 * m + 5)));
}

Krylov::~Krylov() { if (hpin) cudaFreeHost(hpin); }

double Krylov::norm(const double *a) {
    cudaStream_t s = ctx->stream;
    { ProfScope ps_(PROF_GMRES); (count_launch(), k_dot<<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, a, a, part.ptr)); }
    { ProfScope ps_(PROF_GMRES); (count_launch(), k_normalize<<<1, RED_THREADS, 0, s>>>(0, part.ptr, nullptr, nullptr, hcol.ptr, 0)); }
    IBIM_CHECK_LAUNCH();
    IBIM_CUDA(cudaMemcpyAsync(hpin, hcol.ptr, sizeof(double), cudaMemcpyDeviceToHost, s));
    IBIM_CUDA(cudaStreamSynchronize(s));
    return hpin[0];
}

// Restarted GMRES(m) of gmres.cpp:50-164 on the device.  x (in/out) and b are device vectors of
// length n.  `x_is_zero` skips the initial A x (it is exactly zero for a linear operator).
int Krylov::solve(const std::function<void(const double *, double *)> &A, double *x, const double *b, int max_iter,
                  double tol, bool x_is_zero, GmresStats &st) {
    cudaStream_t s = ctx->stream;
    const int eg = ew_grid(ctx, n);
    double normb = norm(b);
    if (x_is_zero) {
        IBIM_CUDA(cudaMemcpyAsync(r.ptr, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    } else {
        A(x, w.ptr);
        st.matvecs++;
        (count_launch(), k_sub<<<eg, 256, 0, s>>>(n, b, w.ptr, r.ptr));
        IBIM_CHECK_LAUNCH();
    }
    double beta = norm(r.ptr);
    if (normb == 0.0) normb = 1;
    double resid = beta / normb;
    st.residual = resid;
    if (resid <= tol) return 0;
    std::vector<double> H((size_t)(m + 1) * (m + 1), 0.), sv(m + 1), cs(m + 1), sn(m + 1), y(m + 1);
    auto Hm = [&](int i, int j) -> double & { return H[(size_t)i * (m + 1) + j]; };
    const int regs = arnoldi_regs(ctx, n);
    unsigned *const ran_out = reinterpret_cast<unsigned *>(hpin + 2 * m + 4);
    int j = 1, i = 0;
    auto update = [&](int k) {
        // back substitution (gmres.cpp:9-21), then x += V y on the device
        if (k < 0) return;
        for (int q = 0; q <= k; ++q) y[q] = sv[q];
        for (int q = k; q >= 0; --q) {
            y[q] /= Hm(q, q);
            for (int l = q - 1; l >= 0; --l) y[l] -= Hm(l, q) * y[q];
        }
        std::copy(y.begin(), y.begin() + k + 1, hpin + m + 2);
        IBIM_CUDA(cudaMemcpyAsync(ydev.ptr, hpin + m + 2, sizeof(double) * (k + 1), cudaMemcpyHostToDevice, s));
        { ProfScope ps_(PROF_GMRES); (count_launch(), k_update<<<eg, 256, 0, s>>>(n, k + 1, ydev.ptr, V.ptr, x)); }
        IBIM_CHECK_LAUNCH();
        if (regs) IBIM_CUDA(cudaMemcpyAsync(ran_out, bar.ptr + 1, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        IBIM_CUDA(cudaStreamSynchronize(s));  // hpin reused next step
        if (regs && *ran_out) throw Error(IBIM_ERR_LIMIT, "Arnoldi step: a wait of its grid exceeded its bound");
    };
    while (j <= max_iter) {
        // v0 = r / beta
        { ProfScope ps_(PROF_GMRES); (count_launch(), k_normalize<<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, part.ptr, r.ptr, V.ptr, hcol.ptr, 0)); }
        std::fill(sv.begin(), sv.end(), 0.);
        sv[0] = beta;
        for (i = 0; i < m && j <= max_iter; i++, j++) {
            double *vi = V.ptr + (size_t)i * n;
            A(vi, w.ptr);
            st.matvecs++;
            st.iters++;
            if (regs) {
                ProfScope ps_(PROF_GMRES);
                const double *wp = w.ptr;
                double *Vp = V.ptr, *pp = part.ptr, *hp = hcol.ptr;
                unsigned *bp = bar.ptr;
                void *args[] = {&n, &i, &wp, &Vp, &pp, &hp, &bp, &arrived};
                const int grid = std::min(RED_BLOCKS / ARN_LANES, div_up(n, ARN_THREADS));
                count_launch();
                IBIM_CUDA(cudaLaunchCooperativeKernel(arnoldi_kernel(regs), dim3(grid), dim3(ARN_THREADS), args, 0, s));
                arrived += (unsigned)((i + 2) * grid);
            } else {
                double *pa = part.ptr, *pb = part.ptr + RED_BLOCKS;
                { ProfScope ps_(PROF_GMRES); (count_launch(), k_dot<<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, w.ptr, V.ptr, pa)); }
                for (int k = 1; k <= i + 1; ++k) {
                    const double *vnext = k <= i ? V.ptr + (size_t)k * n : nullptr;
                    { ProfScope ps_(PROF_GMRES); (count_launch(), k_mgs<<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, pa, w.ptr, V.ptr + (size_t)(k - 1) * n, vnext, pb,
                                                             hcol.ptr, k - 1)); }
                    std::swap(pa, pb);
                }
                { ProfScope ps_(PROF_GMRES); (count_launch(), k_normalize<<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, pa, w.ptr, V.ptr + (size_t)(i + 1) * n, hcol.ptr, i + 1)); }
            }
            IBIM_CHECK_LAUNCH();
            IBIM_CUDA(cudaMemcpyAsync(hpin, hcol.ptr, sizeof(double) * (i + 2), cudaMemcpyDeviceToHost, s));
            IBIM_CUDA(cudaStreamSynchronize(s));
            for (int k = 0; k <= i + 1; ++k) Hm(k, i) = hpin[k];
            for (int k = 0; k < i; ++k) apply_rot(Hm(k, i), Hm(k + 1, i), cs[k], sn[k]);
            gen_rot(Hm(i, i), Hm(i + 1, i), cs[i], sn[i]);
            apply_rot(Hm(i, i), Hm(i + 1, i), cs[i], sn[i]);
            apply_rot(sv[i], sv[i + 1], cs[i], sn[i]);
            resid = std::fabs(sv[i + 1]) / normb;
            st.history.push_back(resid);
            if (resid < tol) {
                update(i);
                st.residual = resid;
                return 0;
            }
        }
        update(i - 1);
        A(x, w.ptr);
        st.matvecs++;
        (count_launch(), k_sub<<<eg, 256, 0, s>>>(n, b, w.ptr, r.ptr));
        IBIM_CHECK_LAUNCH();
        // ||r||: partials of <r, r> land in part[0..) for the k_normalize of the next cycle
        { ProfScope ps_(PROF_GMRES); (count_launch(), k_dot<<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, r.ptr, r.ptr, part.ptr)); }
        { ProfScope ps_(PROF_GMRES); (count_launch(), k_normalize<<<1, RED_THREADS, 0, s>>>(0, part.ptr, nullptr, nullptr, hcol.ptr, 0)); }
        IBIM_CHECK_LAUNCH();
        IBIM_CUDA(cudaMemcpyAsync(hpin, hcol.ptr, sizeof(double), cudaMemcpyDeviceToHost, s));
        IBIM_CUDA(cudaStreamSynchronize(s));
        beta = hpin[0];
        resid = beta / normb;
        st.residual = resid;
        if (resid < tol) return 0;
    }
    return 1;
}

// The first k_normalize of each cycle reads the <r, r> partials from part[0..RED_BLOCKS).
// norm() leaves them there; so does the restart above.

// ---------------------------------------------------------------------------------------
// Whole BIE solve on a plan: RHS, GMRES (FP64 or mixed with FP64 refinement), polarize, energy
// ---------------------------------------------------------------------------------------

void electric_solve(Plan &P, const ibim_kernel_params &kp, const double *atoms4_dev, const double *charges_host,
                    int natoms, int restart, int maxiter, double tol, int precision, double *x_tree_out,
                    std::vector<double> *atom_pot, ibim_result &res, const double *b_tube) {
    Ctx *c = P.ctx;
    cudaStream_t s = c->stream;
    const long n2 = 2 * P.ns;
    DevBuf<double> b, x;
    b.alloc(n2, s);
    x.alloc(n2, s);
    x.zero();
    Timer tm(s);
    if (b_tube) {
        // right-hand side computed in tube order beforehand: into tree order
        permute(c, P.ns, P.src_perm.ptr, b_tube, b.ptr, false);
        permute(c, P.ns, P.src_perm.ptr, b_tube + P.ns, b.ptr + P.ns, false);
    } else {
        bie_rhs(P, kp, atoms4_dev, natoms, b.ptr);
    }
    Krylov K(c, n2, std::max(1, std::min(restart, 250)));
    GmresStats st;
    int status = 1;
    const bool plain = precision != IBIM_PRECISION_MIXED;  // FP64, or FP64 with tensor-core M2L
    if (plain) {
        auto A = [&](const double *in, double *out) { bie_matvec(P, kp, in, out, precision); };
        status = K.solve(A, x.ptr, b.ptr, maxiter, tol, true, st);
        res.matvecs_fp64 = st.matvecs;
        res.refinements = 0;
    } else {
        // FP64 iterative refinement around the mixed-precision GMRES
        auto A32 = [&](const double *in, double *out) { bie_matvec(P, kp, in, out, IBIM_PRECISION_MIXED); };
        // residual operator: FP64 with the V-list M2L as exact digit products on the tensor cores
        // (IBIM_RESIDUAL_M2L=fp64 selects the FP64-pipe M2L, for comparison)
        const char *rm = std::getenv("IBIM_RESIDUAL_M2L");
        const int res_prec = (rm && std::string(rm) == "fp64") ? IBIM_PRECISION_FP64 : IBIM_PRECISION_FP64_TC;
        auto A64 = [&](const double *in, double *out) { bie_matvec(P, kp, in, out, res_prec); };
        DevBuf<double> r, d;
        r.alloc(n2, s);
        d.alloc(n2, s);
        IBIM_CUDA(cudaMemcpyAsync(r.ptr, b.ptr, sizeof(double) * n2, cudaMemcpyDeviceToDevice, s));
        const double normb = K.norm(b.ptr);
        int fp64 = 0, outer = 0, left = maxiter;
        double rel = 1.0;
        for (outer = 0; outer < 8 && left > 0; ++outer) {
            d.zero();
            GmresStats si;
            // inner tolerance relative to ||r||: 0.7 of the outer target (the rest is left for the gap
            // between the mixed and the FP64-class operator, small once both decide the near-field
            // cutoff alike), above the FP32 noise floor.  IBIM_IR_FACTOR in (0, 1) replaces the 0.7.
            static const double factor = [] {
                const char *v = std::getenv("IBIM_IR_FACTOR");
                const double f = v ? std::atof(v) : 0.7;
                return f > 0.0 && f < 1.0 ? f : 0.7;
            }();
            const double inner = std::min(0.5, std::max(factor * tol / rel, 3e-7));
            K.solve(A32, d.ptr, r.ptr, left, inner, true, si);
            trace_mark("electric: inner gmres");
            st.iters += si.iters;
            st.matvecs += si.matvecs;
            left -= si.iters;
            (count_launch(), k_axpy<<<ew_grid(c, n2), 256, 0, s>>>(n2, 1.0, d.ptr, x.ptr));
            A64(x.ptr, K.w.ptr);
            fp64++;
            (count_launch(), k_sub<<<ew_grid(c, n2), 256, 0, s>>>(n2, b.ptr, K.w.ptr, r.ptr));
            IBIM_CHECK_LAUNCH();
            rel = K.norm(r.ptr) / (normb == 0 ? 1 : normb);
            trace_mark("electric: fp64-class residual");
            st.history.push_back(rel);
            if (rel < tol) break;
        }
        st.residual = rel;
        status = rel < tol ? 0 : 1;
        res.matvecs_fp64 = fp64;
        res.refinements = outer + (outer < 8 ? 1 : 0);
    }
    res.gmres_iters = st.iters;
    res.matvecs = st.matvecs + (plain ? 0 : res.matvecs_fp64);
    res.gmres_status = status;
    res.residual = st.residual;
    res.t_solve_ms = tm.ms();
    // polarizeMap + energy (electric.cpp:442-505): targets = atoms (target set 1)
    Timer te(s);
    if (natoms > 0 && P.targets.size() > 1) {
        TargetSet &A = *P.targets[1];
        (count_launch(), k_densities<<<ew_grid(c, P.ns), 256, 0, s>>>(P.ns, x.ptr, P.snx.ptr, P.sny.ptr, P.snz.ptr, P.sw.ptr,
                                                      P.dens4.ptr));
        IBIM_CHECK_LAUNCH();
        fmm_run(P, 1, kp, P.dens4.ptr, A.out4.ptr, precision);
        std::vector<double> F(A.nt);
        A.out4.download(F.data(), A.nt);
        IBIM_CUDA(cudaStreamSynchronize(s));
        std::vector<double> pot(natoms, 0.);
        for (long q = 0; q < A.nt; ++q) pot[A.perm[q]] = -F[q];  // ret2 - (ret1x + ret1y + ret1z)
        double E = 0.;
        for (int a = 0; a < natoms; ++a) E += pot[a] * charges_host[a];
        res.energy = 0.5 * E;
        if (atom_pot) *atom_pot = pot;
    }
    res.t_energy_ms = te.ms();
    trace_mark("electric: energy");
    if (m2l_tc_error(P)) throw Error(IBIM_ERR_LIMIT, "tensor-core M2L: an MMA completion wait exceeded its bound");
    if (x_tree_out) IBIM_CUDA(cudaMemcpyAsync(x_tree_out, x.ptr, sizeof(double) * n2, cudaMemcpyDeviceToDevice, s));
    IBIM_CUDA(cudaStreamSynchronize(s));
}

}  // namespace ibim
