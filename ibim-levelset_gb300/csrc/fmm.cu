// Black-box Chebyshev FMM on the GPU (sm_103a), FP64 path.
//
// Replaces bbfmm::kernel (bbfmm.h:200-624) for the reference's BIE kernel set.  One pass
// computes the fused 4-density -> 4-field operator (the 16 scalar FMMs of one matvec,
// electric.cpp:333-367, share one tree and one set of Chebyshev operators, so their sum is
// one FMM with a 4x4 kernel block):
//   inputs  m_x, m_y, m_z = phi n w,  psi = dphi w        (electric.cpp:324-329)
//   outputs F   = K1 . m - K2 psi                           (-> out1, electric.cpp:382)
//           G_a = sum_b H_ab m_b - K4_a psi, H = K3 block   (-> n . G = tmp1 - tmp2, :372-383)
// Same approximation as the reference: Chebyshev order p, leaf P2M/L2P through the tensor
// interpolant S_p (bbfmm.h:392-433), M2M/L2L through the 8 Kronecker operators (:305-367),
// M2L for V and X lists with the kernel at Chebyshev node pairs (:547-561), direct U and W
// lists (:577-595).
//
// Data layout in HBM: points SoA in tree order (each node owns a contiguous range);
// multipole / local coefficients per node as [4][p^3] with index z*p^2 + y*p + x.
// V-list M2L: the kernel at Chebyshev node pairs depends only on (level, source - target
// lattice offset), so those (4p^3)^2 operators are built once per plan and applied as a
// batched dense contraction (pairs grouped by operator).

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <unordered_map>
#include <tuple>

#include <omp.h>

#include "fmm_common.cuh"
#include "fp64_seed.cuh"

namespace ibim {

// ----------------------------------------------------------------------------------------
// Tables
// ----------------------------------------------------------------------------------------

void cheb_tables_host(int p, ChebTables &T) {
    std::memset(&T, 0, sizeof(T));
    T.p = p;
    T.R = p * p * p;
    for (int i = 0; i < p; ++i) T.cheb[i] = -std::cos((i + 0.5) * M_PI / p);
    auto poly = [&](double x, double *out) {
        out[0] = 1.0;
        if (p > 1) out[1] = x;
        for (int k = 2; k < p; ++k) out[k] = 2.0 * x * out[k - 1] - out[k - 2];
    };
    for (int m = 0; m < p; ++m) poly(T.cheb[m], T.tnode[m]);
    // parent -> child transfer S[bit][child node][parent node] (bbfmm.h:305-326)
    for (int a = 0; a < 2 * p; ++a) {
        const double x = a < p ? 0.5 * T.cheb[a] - 0.5 : 0.5 * T.cheb[a - p] + 0.5;
        double tx[MAXP];
        poly(x, tx);
        for (int m = 0; m < p; ++m) {
            double s = 0.;
            for (int k = 0; k < p; ++k) s += tx[k] * T.tnode[m][k];
            T.S[a / p][a % p][m] = (-1.0 + 2.0 * s) * (1.0 / p);
        }
    }
}

// ----------------------------------------------------------------------------------------
// FP64 kernels
// ----------------------------------------------------------------------------------------

namespace {

// Build the M2L operators: op (target level, source level, centre offset D in target half-widths)
// -> K[col * 4R + row], row = out * R + ct, col = in * R + cs,
// entry = block(src_cheb(cs) - tgt_cheb(ct))[out][in], node positions D r_t + r_s cheb - r_t cheb.
// V operators (same level, D = 2 o) and X operators (coarser source leaf) share the layout.
__device__ __forceinline__ void op_geometry(const int *keys, int op, const double *root_r, double rt[3], double rs[3],
                                            int D[3]) {
    const int lt = keys[5 * op], ls = keys[5 * op + 1];
    for (int a = 0; a < 3; ++a) {
        double vt = root_r[a], vs = root_r[a];
        for (int l = 0; l < lt; ++l) vt *= 0.5;
        for (int l = 0; l < ls; ++l) vs *= 0.5;
        rt[a] = vt;
        rs[a] = vs;
        D[a] = keys[5 * op + 2 + a];
    }
}

// One entry of the block (entry = 4 out + in) gives R x R operators K[cs * R + ct].  The FP64 pipe bounds the
// evaluation, so a class of mirror images is evaluated once (Mirror) by classes blockIdx.y of cls, ord; the members
// lie at their own places, or from pos0 on in the order of ord.
// 1,405 operators of order 5 with their digit images: 7.3 -> 3.7 ms.
__global__ void k_make_ops64(const ChebTables *__restrict__ tab, const int *__restrict__ keys,
                             const double *__restrict__ root_r, KParams kp, int entry, const int *__restrict__ cls,
                             const int *__restrict__ ord, int pos0, double *ops) {
    const ChebTables &T = *tab;
    const int m0 = cls[blockIdx.y], m1 = cls[blockIdx.y + 1];
    const int p = T.p, R = T.R, n4 = 4 * R;
    double rt[3], rs[3];
    int D[3];
    op_geometry(keys, ord[m0], root_r, rt, rs, D);
    // consecutive threads take consecutive target nodes ct, so each output row is written by
    // contiguous 8-byte stores
    const long pair = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (pair >= (long)R * R) return;
    const int cs = (int)(pair / R), ct = (int)(pair % R);
    const int ti[3] = {ct % p, (ct / p) % p, ct / (p * p)};
    const int si[3] = {cs % p, (cs / p) % p, cs / (p * p)};
    double d[3];
    for (int a = 0; a < 3; ++a) d[a] = (abs(D[a]) * rt[a] + rs[a] * T.cheb[si[a]]) - rt[a] * T.cheb[ti[a]];
    double b[16];
    kblock64(kp, d[0], d[1], d[2], b);
    for (int m = m0; m < m1; ++m) {
        const Mirror M(keys + 5 * ord[m], p, ti, si);
        const long at = pos0 < 0 ? ord[m] : m - pos0;
        if (entry != ENTRY_BLOCK) {
            double v = b[0];
#pragma unroll
            for (int i = 1; i < 16; ++i) v = i == entry ? b[i] : v;
            ops[at * R * R + (long)M.cs * R + M.ct] = M.flip(entry >> 2, entry & 3) ? -v : v;
            continue;
        }
        double *K = ops + at * n4 * n4;
#pragma unroll
        for (int o = 0; o < 4; ++o)
#pragma unroll
            for (int in = 0; in < 4; ++in)
                K[(long)(in * R + M.cs) * n4 + (o * R + M.ct)] = M.flip(o, in) ? -b[o * 4 + in] : b[o * 4 + in];
    }
}

// V-list M2L as a batched contraction: chunk = (op, first pair, count <= M2L_CH); every
// thread owns rows r = tid + 256 q of the 4R outputs for all pairs of the chunk.
constexpr int M2L_CH = 8;
__global__ void __launch_bounds__(256) k_m2l_v64(int n4, const int *__restrict__ chunks, const int *__restrict__ vsrc,
                                                 const int *__restrict__ vtgt, const double *__restrict__ ops,
                                                 const double *__restrict__ mult, double *local) {
    extern __shared__ double Ms[];  // [M2L_CH][n4]
    const int op = chunks[3 * blockIdx.x], b = chunks[3 * blockIdx.x + 1], cnt = chunks[3 * blockIdx.x + 2];
    for (int j = 0; j < cnt; ++j) {
        const double *src = mult + (long)vsrc[b + j] * n4;
        for (int o = threadIdx.x; o < n4; o += blockDim.x) Ms[j * n4 + o] = src[o];
    }
    __syncthreads();
    const double *K = ops + (long)op * n4 * n4;
    constexpr int MAXQ = 8;  // n4 <= 2048
    double acc[MAXQ][M2L_CH];
#pragma unroll
    for (int q = 0; q < MAXQ; ++q)
#pragma unroll
        for (int j = 0; j < M2L_CH; ++j) acc[q][j] = 0.;
    const int nq = (n4 + 255) / 256;
    for (int col = 0; col < n4; ++col) {
        const double *Kc = K + (long)col * n4;
#pragma unroll
        for (int q = 0; q < MAXQ; ++q) {
            if (q >= nq) break;
            const int row = threadIdx.x + 256 * q;
            const double a = row < n4 ? __ldg(Kc + row) : 0.;
#pragma unroll
            for (int j = 0; j < M2L_CH; ++j) acc[q][j] += a * Ms[j * n4 + col];
        }
    }
#pragma unroll
    for (int q = 0; q < MAXQ; ++q) {
        if (q >= nq) break;
        const int row = threadIdx.x + 256 * q;
        if (row >= n4) continue;
#pragma unroll
        for (int j = 0; j < M2L_CH; ++j)
            if (j < cnt) atomicAdd(local + (long)vtgt[b + j] * n4 + row, acc[q][j]);
    }
}

// X-list M2L (bbfmm.h:556-560): coarser leaf -> node, kernel evaluated on the fly.
__global__ void __launch_bounds__(128) k_m2l_x64(const ChebTables *__restrict__ tab, KParams kp,
                                                 const int *__restrict__ xsrc, const int *__restrict__ xtgt,
                                                 const double *__restrict__ ctr, const double *__restrict__ rad,
                                                 const double *__restrict__ mult, double *local) {
    __shared__ ChebTables T;
    __shared__ double M[4 * MAXR];
    __shared__ double sp[3][MAXP], tp[3][MAXP];
    for (int t = threadIdx.x; t < (int)(sizeof(ChebTables) / 8); t += blockDim.x)
        reinterpret_cast<double *>(&T)[t] = reinterpret_cast<const double *>(tab)[t];
    __syncthreads();
    const int s = xsrc[blockIdx.x], t = xtgt[blockIdx.x];
    const int p = T.p, R = T.R;
    for (int o = threadIdx.x; o < 4 * R; o += blockDim.x) M[o] = mult[(long)s * 4 * R + o];
    if (threadIdx.x < 3 * p) {
        const int a = threadIdx.x / p, m = threadIdx.x % p;
        sp[a][m] = ctr[3 * s + a] + rad[3 * s + a] * T.cheb[m];
        tp[a][m] = ctr[3 * t + a] + rad[3 * t + a] * T.cheb[m];
    }
    __syncthreads();
    for (int ct = threadIdx.x; ct < R; ct += blockDim.x) {
        const double tx = tp[0][ct % p], ty = tp[1][(ct / p) % p], tz = tp[2][ct / (p * p)];
        double acc[4] = {0., 0., 0., 0.};
        for (int cs = 0; cs < R; ++cs) {
            double b[16];
            kblock64(kp, sp[0][cs % p] - tx, sp[1][(cs / p) % p] - ty, sp[2][cs / (p * p)] - tz, b);
#pragma unroll
            for (int o = 0; o < 4; ++o)
#pragma unroll
                for (int in = 0; in < 4; ++in) acc[o] += b[o * 4 + in] * M[in * R + cs];
        }
        for (int o = 0; o < 4; ++o) atomicAdd(local + (long)t * 4 * R + o * R + ct, acc[o]);
    }
}

// Near field + L2P for one target leaf per block (downPass leaf, bbfmm.h:571-609): U and W
// lists direct (source ranges in tree order), then the local expansion at the targets.
// Threads = targets x source phases; sources staged in shared memory tiles.
//
// Bound by GB300's narrow FP64 pipe (2 lanes a cycle per SM: 16 cycles a warp instruction, whatever
// else the SM does), so the count of FP64 instructions a pair is the kernel's time.  near64_pair
// takes 42 (20 without screening) where the formulas as written took about 103: seeds, their refinement,
// rounding and comparisons on the integer and FP32 pipes, a 512-entry table and a polynomial of degree 4, half of
// it in FP32, for the exponential, and the constant factors applied once per target instead of
// once per pair.  16 warps a SM keep the pipe busy; two CTAs of 14 KB leave the rest of the SM to
// the tensor-core M2L that runs beside it.  On a 2,000-atom protein (5.2e8 pairs): 82 -> 43 ms alone
// (42 instructions take 35 ms; 51, with a cubic step for 1 / r and all of the polynomial in FP64, 49 ms), 46 ms
// beside the M2L.
constexpr int NEAR_T = 256, NEAR_TILE = 128, NEAR_CPS = 2;  // threads, sources a tile, CTAs a SM
constexpr int NEAR_EXP = 512;                               // steps of 2^-x in the table
enum { NEAR_GENERAL = 0, NEAR_YUKAWA = 1, NEAR_LAPLACE = 2 };

struct Near64K {
    double vr2, eps, ieps, kappa, kappa2, kl;  // kl = kappa log2 e
    double sk, k2c;                    // k3f / q4pi; k2in k3f / q4pi^2 (the cutoff's K2 in A0's units)
    double psi_f, f0, fg;              // staged psi = psi psi_f; F = f0 A0, G = fg A
    float klt;                         // kl NEAR_EXP
    KParams kp;
};

Near64K make_near64(const KParams &k) {
    Near64K n{};
    n.kp = k;
    n.vr2 = k.vr2;
    n.eps = k.eps;
    n.ieps = k.ieps;
    n.kappa = k.kappa;
    n.kappa2 = k.kappa * k.kappa;
    n.kl = k.kappa * 1.4426950408889634074;
    n.sk = k.k3f / k.q4pi;
    n.psi_f = k.q4pi / k.k3f;
    n.k2c = k.k2in * (n.sk / k.q4pi);
    n.f0 = k.q4pi;
    n.fg = k.k3f;
    n.klt = (float)(n.kl * NEAR_EXP);
    return n;
}

__device__ __forceinline__ bool nonfinite64(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// FP32 value of a double below 2^127 in magnitude by its bits (truncated; below 2^-126: 0).
__device__ __forceinline__ float near64_f32(double v) {
    const unsigned hi = __double2hiint(v), mag = hi & 0x7fffffff;
    if (mag < 0x38100000) return 0.f;
    return __uint_as_float((hi & 0x80000000) | ((mag - 0x38000000) << 3) | ((unsigned)__double2loint(v) >> 29));
}
// The double equal to a non-negative normal float (0 becomes 2^-127).
__device__ __forceinline__ double near64_f64(float v) {
    const int b = __float_as_int(v);
    return __hiloint2double((b >> 3) + 0x38000000, b << 29);
}

// 1 / sqrt(d2) for normal d2 > 0 in three FP64 instructions, and sqrt(d2) to FP32 (at most 2^121): the seed y of
// 2^-44, y + y e with e = (1 - d2 y^2) / 2.
__device__ __forceinline__ double near64_rsqrt(double d2, float &rf) {
    const double y = rsqrt_seed(d2, rf);
    return fma(y, fma(d2 * y, -half_of(y), 0.5), y);
}

// t = kappa r and e = e^-t = 2^{-n/512} 2^{-g}: n from the FP32 r, g exact, |g| <= 2^-10 (2^-9.7 where e is below
// 2^-900); Taylor to degree 4 (below 2^-59), the two highest coefficients, 2^-34 of the whole, in FP32.
__device__ __forceinline__ void near64_exp(const Near64K &k, const double *__restrict__ e2, double r, float rf, double &t,
                                           double &e) {
    t = k.kappa * r;
    const float xm = fminf(rf * k.klt, 1000.f * NEAR_EXP) + 12582912.f;  // n in the low bits
    const int n = __float_as_int(xm) - 0x4b400000;
    const double g = fma(k.kl, r, -near64_f64((xm - 12582912.f) * (1.f / NEAR_EXP)));
    const float h = fmaf(near64_f32(g), -9.6181291e-3f, 5.5504109e-2f);
    double q = fma(-near64_f64(h), g, 2.4022650695910072e-1);
    q = fma(g, q, -6.9314718055994531e-1) * g;
    const double tb = e2[n & (NEAR_EXP - 1)];
    const double ef = fma(tb, q, tb);
    e = n >= 1000 * NEAR_EXP ? 0.0
                             : __hiloint2double(__double2hiint(ef) - ((n / NEAR_EXP) << 20), __double2loint(ef));
}

// One source -> target update of the fused block (kblock64's formulas) for d2 >= vr2, with
// M = d.m / r^3 shared by K1 and K3, psi staged times q4pi / k3f, and the factors q4pi (F) and
// k3f (G) left to the caller.  With u = 1 - e^-t (1 + t): ho / r^2 = kappa^2 e^-t - 3 u / r^2 and hd = u / r^3; 3 u
// serves both, with the dipole also staged a third as large (n).
template <int MODE>
__device__ __forceinline__ void near64_pair(const Near64K &k, const double *__restrict__ e2, double dx, double dy,
                                            double dz, double m0, double m1, double m2, double psi, double n0, double n1,
                                            double n2, double acc[4]) {
    const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
    // both non-negative: the order of the bits is the order of the values
    if (__double_as_longlong(d2) < __double_as_longlong(k.vr2)) {
        if (MODE == NEAR_YUKAWA) acc[0] = fma(-k.k2c, psi, acc[0]);
        return;
    }
    float rf;
    const double ir = near64_rsqrt(d2, rf);
    const double ir2 = ir * ir, ir3 = ir2 * ir;
    const double M = fma(dx, m0, fma(dy, m1, dz * m2)) * ir3;
    const double w = ir3 * psi;
    if (MODE == NEAR_LAPLACE) {  // e = 1: K2 = K3 = 0
        acc[0] += M;
        acc[1] = fma(dx, w, acc[1]);
        acc[2] = fma(dy, w, acc[2]);
        acc[3] = fma(dz, w, acc[3]);
        return;
    }
    double t, e;
    near64_exp(k, e2, d2 * ir, rf, t, e);
    const double et1 = fma(e, t, e);
    acc[0] = fma(fma(k.eps, et1, -1.0), M, acc[0]);
    acc[0] = fma(-(fma(-k.sk, e, k.sk) * ir), psi, acc[0]);
    const double u3 = fma(-3.0, et1, 3.0);
    const double cm = fma(fma(-u3, ir2, e * k.kappa2), M, -(fma(-k.ieps, et1, 1.0) * w));
    const double hd3 = u3 * ir3;
    acc[1] = fma(dx, cm, fma(hd3, n0, acc[1]));
    acc[2] = fma(dy, cm, fma(hd3, n1, acc[2]));
    acc[3] = fma(dz, cm, fma(hd3, n2, acc[3]));
}

// One scalar kernel's update, an entry of the block above by the same steps (22 to 26 FP64 instructions
// screened, 14 not): a and b are the axes of the dipole (K1, K3) and of the gradient (K3, K4).
enum { NEAR_BLOCK = 0, NEAR_K1 = 1, NEAR_K2 = 2, NEAR_K3 = 3, NEAR_K4 = 4 };
template <int MODE, int KIND>
__device__ __forceinline__ double near64_one(const Near64K &k, const double *__restrict__ e2, double dx, double dy,
                                             double dz, int a, int b, double m, double acc) {
    const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const double da = a == 0 ? dx : (a == 1 ? dy : dz), db = b == 0 ? dx : (b == 1 ? dy : dz);
    if (MODE == NEAR_GENERAL) {
        if (d2 < k.vr2) return KIND == NEAR_K2 ? fma(-k.kp.k2in, m, acc) : acc;
        double c1, c4, k2, hd, ho;
        radial64(k.kp, d2, c1, c4, k2, hd, ho);
        if (KIND == NEAR_K1) return fma(c1, da * m, acc);
        if (KIND == NEAR_K2) return fma(-k2, m, acc);
        if (KIND == NEAR_K3) return fma(db, ho * (da * m), a == b ? fma(hd, m, acc) : acc);
        return fma(db, -c4 * m, acc);
    }
    if (MODE == NEAR_LAPLACE && (KIND == NEAR_K2 || KIND == NEAR_K3)) return acc;
    if (__double_as_longlong(d2) < __double_as_longlong(k.vr2)) return KIND == NEAR_K2 ? fma(-k.k2c, m, acc) : acc;
    float rf;
    const double ir = near64_rsqrt(d2, rf);
    const double ir2 = ir * ir, ir3 = ir2 * ir;
    if (MODE == NEAR_LAPLACE) return fma((KIND == NEAR_K1 ? da : db) * m, ir3, acc);
    double t, e;
    near64_exp(k, e2, d2 * ir, rf, t, e);
    if (KIND == NEAR_K2) return fma(-(fma(-k.sk, e, k.sk) * ir), m, acc);
    const double et1 = fma(e, t, e);
    if (KIND == NEAR_K1) return fma(fma(k.eps, et1, -1.0), (da * m) * ir3, acc);
    if (KIND == NEAR_K4) return fma(db, -fma(-k.ieps, et1, 1.0) * (ir3 * m), acc);
    const double u = 1.0 - et1, mi3 = m * ir3;
    if (a == b) acc = fma(u, mi3, acc);
    return fma(db * da, fma(-3.0 * u, ir2, e * k.kappa2) * mi3, acc);
}

template <int MODE, int KIND>
__global__ void __launch_bounds__(NEAR_T, 3)  // 80 registers: two CTAs leave the M2L its own
    k_near64(const ChebTables *__restrict__ tab, const double *__restrict__ etab, Near64K kp, const int4 *__restrict__ segs,
             const int *__restrict__ near_range, const int *__restrict__ tb_, const int *__restrict__ te_,
             const double *__restrict__ ctr, const double *__restrict__ rad, const double *__restrict__ sx,
             const double *__restrict__ sy, const double *__restrict__ sz, const double *__restrict__ dens, long ns,
             const double *__restrict__ tx, const double *__restrict__ ty, const double *__restrict__ tz, long nt,
             const double *__restrict__ local, double *out, int l2p_mask, int nseg, int *next, int ax_in, int ax_out) {
    constexpr int NC = KIND == NEAR_BLOCK ? 4 : 1;
    constexpr bool FG = KIND == NEAR_K1 || KIND == NEAR_K2;  // the one output is F
    // Without screening K2 and K3 are zero and their terms are left out, but for NaN and infinite densities
    constexpr bool ZEROS = MODE == NEAR_LAPLACE && (NC == 4 || KIND == NEAR_K2 || KIND == NEAR_K3);
    // x y | z m_x | m_y m_z | psi n_x | n_y n_z (n = m / 3), one kernel: x y | z m
    __shared__ double2 S[NEAR_TILE][NC == 4 ? 5 : 2];
    __shared__ double e2[MODE == NEAR_YUKAWA ? NEAR_EXP : 1];  // 2^(-j / 512)
    __shared__ int cur;
    double(*red)[NC] = reinterpret_cast<double(*)[NC]>(S);  // [NEAR_T][NC], once the tiles are done
    static_assert(sizeof(S) >= sizeof(double) * NC * NEAR_T, "reduction scratch");
    if (MODE == NEAR_YUKAWA)
        for (int i = threadIdx.x; i < NEAR_EXP; i += NEAR_T) e2[i] = etab[i];
    const double psi_f = MODE == NEAR_GENERAL ? 1.0 : kp.psi_f;
    // with a work counter the CTA takes segments until none is left; without one it does segment blockIdx.x
    for (int it = 0;; ++it) {
        int si;
        if (next) {
            __syncthreads();  // every thread has read the previous segment number
            if (threadIdx.x == 0) cur = atomicAdd(next, 1);
            __syncthreads();
            si = cur;
            if (si >= nseg) break;
        } else {
            if (it > 0) break;
            si = blockIdx.x;
        }
        const int4 sg = segs[si];
        const int leaf = sg.x, r0 = sg.y, r1 = sg.z, mode = sg.w;
        const int tb = tb_[leaf], te = te_[leaf];
        __syncthreads();
        for (int t0 = tb; t0 < te; t0 += NEAR_T) {
            const int nT = min(NEAR_T, te - t0);
            const int nph = NEAR_T / nT;
            const int my_t = threadIdx.x % nT, ph = threadIdx.x / nT;
            const bool active = ph < nph;
            double X = 0, Y = 0, Z = 0;
            if (active) { X = tx[t0 + my_t]; Y = ty[t0 + my_t]; Z = tz[t0 + my_t]; }
            double acc[NC] = {};
            for (int rr = r0; rr < r1; ++rr) {
                const int b = near_range[2 * rr], e = near_range[2 * rr + 1];
                for (int s0 = b; s0 < e; s0 += NEAR_TILE) {
                    const int cnt = min(NEAR_TILE, e - s0);
                    __syncthreads();
                    // two threads a source
                    const int q = threadIdx.x >> 1;
                    bool bad = false;  // (ZEROS) a NaN or an infinity
                    if (q < cnt) {
                        const long i = s0 + q;
                        if constexpr (NC == 1) {
                            if (threadIdx.x & 1) {
                                const double m = dens[i];
                                bad = nonfinite64(m);
                                S[q][1] = make_double2(sz[i], KIND == NEAR_K2 || KIND == NEAR_K4 ? m * psi_f : m);
                            } else
                                S[q][0] = make_double2(sx[i], sy[i]);
                        } else if (threadIdx.x & 1) {
                            const double m1 = dens[ns + i], m2 = dens[2 * ns + i], psi = dens[3 * ns + i];
                            bad = nonfinite64(m1) || nonfinite64(m2) || nonfinite64(psi);
                            S[q][2] = make_double2(m1, m2);
                            S[q][4] = make_double2(m1 * (1.0 / 3.0), m2 * (1.0 / 3.0));
                            S[q][3].x = psi * psi_f;
                        } else {
                            const double m0 = dens[i];
                            bad = nonfinite64(m0);
                            S[q][0] = make_double2(sx[i], sy[i]);
                            S[q][1] = make_double2(sz[i], m0);
                            S[q][3].y = m0 * (1.0 / 3.0);
                        }
                    }
                    if constexpr (ZEROS) bad = __syncthreads_or(bad);
                    else __syncthreads();
                    if (active)
#pragma unroll 2  // two pairs in flight a warp: 50.4 -> 48.1 ms for the electrostatics of 100 atoms
                        for (int q2 = ph; q2 < cnt; q2 += nph) {
                            const double2 a0 = S[q2][0], a1 = S[q2][1];
                            if constexpr (NC == 1) {
                                acc[0] = near64_one<MODE, KIND>(kp, e2, a0.x - X, a0.y - Y, a1.x - Z, ax_in, ax_out, a1.y,
                                                                acc[0]);
                                continue;
                            } else {
                            const double2 a2 = S[q2][2], a3 = S[q2][3], a4 = S[q2][4];
                            if (MODE == NEAR_GENERAL)
                                near_pair64(kp.kp, a0.x - X, a0.y - Y, a1.x - Z, a1.y, a2.x, a2.y, a3.x, acc);
                            else
                                near64_pair<MODE>(kp, e2, a0.x - X, a0.y - Y, a1.x - Z, a1.y, a2.x, a2.y, a3.x, a3.y, a4.x,
                                                  a4.y, acc);
                            }
                        }
                    if constexpr (ZEROS)
                        if (bad && active)  // 0 times them
                            for (int q2 = ph; q2 < cnt; q2 += nph) {
                                const double2 a0 = S[q2][0], a1 = S[q2][1];
                                const double dx = a0.x - X, dy = a0.y - Y, dz = a1.x - Z;
                                const bool inside = fma(dx, dx, fma(dy, dy, dz * dz)) < kp.vr2;
                                if constexpr (NC == 1) {
                                    if (KIND == NEAR_K2 || !inside) acc[0] += 0.0 * a1.y;
                                } else {
                                    acc[0] += 0.0 * S[q2][3].x;
                                    const double dm = fma(dx, a1.y, fma(dy, S[q2][2].x, dz * S[q2][2].y));
                                    if (!inside)
                                        for (int o = 1; o < 4; ++o) acc[o] += 0.0 * dm;
                                }
                            }
                }
            }
            if (MODE != NEAR_GENERAL) {
                // without screening the pairs carry c1 = eps - 1 and -c4 = 1/eps - 1 here
                if (NC == 4 || FG) acc[0] *= MODE == NEAR_LAPLACE ? kp.f0 * (kp.eps - 1.0) : kp.f0;
                for (int o = NC == 4 || FG ? 1 : 0; o < NC; ++o) acc[o] *= MODE == NEAR_LAPLACE ? kp.fg * (kp.ieps - 1.0) : kp.fg;
            }
            __syncthreads();  // every thread is done with the last tile
            for (int o = 0; o < NC; ++o) red[threadIdx.x][o] = acc[o];
            __syncthreads();
            if (threadIdx.x < nT) {
                double f[NC] = {};
                for (int q = 0; q < nph; ++q)
                    for (int o = 0; o < NC; ++o) f[o] += red[threadIdx.x + q * nT][o];
                // L2P (bbfmm.h:600): local expansion at the target, by the leaf's first segment
                double l2p[NC] = {};
                if (mode & l2p_mask & 1) {
                    const ChebTables &T = *tab;
                    double Sp[3][MAXP];
                    const double xyz[3] = {X, Y, Z};
                    for (int a = 0; a < 3; ++a) interp1(T, (xyz[a] - ctr[3 * leaf + a]) / rad[3 * leaf + a], Sp[a]);
                    const int p = T.p, R = T.R;
                    const double *L = local + (long)leaf * NC * R;
                    for (int c = 0; c < R; ++c) {
                        const double w = Sp[0][c % p] * Sp[1][(c / p) % p] * Sp[2][c / (p * p)];
                        for (int o = 0; o < NC; ++o) l2p[o] += w * L[o * R + c];
                    }
                }
                for (int o = 0; o < NC; ++o) {
                    double *dst = out + o * nt + t0 + threadIdx.x;
                    if (mode & 2) atomicAdd(dst, f[o] + l2p[o]);
                    else *dst = f[o] + l2p[o];
                }
            }
            __syncthreads();
        }
    }
}

using Near64Fn = decltype(&k_near64<NEAR_YUKAWA, NEAR_BLOCK>);
template <int KIND> Near64Fn near64_mode(int mode) {
    return mode == NEAR_YUKAWA ? k_near64<NEAR_YUKAWA, KIND>
                               : (mode == NEAR_LAPLACE ? k_near64<NEAR_LAPLACE, KIND> : k_near64<NEAR_GENERAL, KIND>);
}
Near64Fn near64_kernel(int mode, int kind) {
    switch (kind) {
        case NEAR_K1: return near64_mode<NEAR_K1>(mode);
        case NEAR_K2: return near64_mode<NEAR_K2>(mode);
        case NEAR_K3: return near64_mode<NEAR_K3>(mode);
        case NEAR_K4: return near64_mode<NEAR_K4>(mode);
        default: return near64_mode<NEAR_BLOCK>(mode);
    }
}

void near64_side_by_side(std::atomic<uint64_t> &done) {
    side_by_side(done, {
#define NEAR64_MODES(K) \
    (const void *)k_near64<NEAR_GENERAL, K>, (const void *)k_near64<NEAR_YUKAWA, K>, (const void *)k_near64<NEAR_LAPLACE, K>
                           NEAR64_MODES(NEAR_BLOCK), NEAR64_MODES(NEAR_K1), NEAR64_MODES(NEAR_K2), NEAR64_MODES(NEAR_K3),
                           NEAR64_MODES(NEAR_K4)
#undef NEAR64_MODES
                       });
}

}  // namespace

// ----------------------------------------------------------------------------------------
// Plan
// ----------------------------------------------------------------------------------------

namespace {
__global__ void k_gather(long n, const int *__restrict__ perm, const double *__restrict__ a, double *b, double scale) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        b[i] = a[perm[i]] * scale;
}

void up_int(DevBuf<int> &b, const std::vector<int> &v, cudaStream_t s) {
    b.alloc(std::max<size_t>(1, v.size()), s);
    b.upload(v.data(), v.size());
}
}  // namespace

void plan_gather(Ctx *c, long n, const int *perm, const double *a, double *b, double scale) {
    if (n <= 0) return;
    (count_launch(), k_gather<<<(int)std::min<long>(4L * c->num_sms, div_up(n, 256)), 256, 0, c->stream>>>(n, perm, a, b, scale));
    IBIM_CHECK_LAUNCH();
}


bool near_segments(const std::vector<int> &tl, const std::vector<int> &nt, std::vector<int> &ptr,
                   std::vector<int> &rng, bool split_long, std::vector<int> &seg, long max_pairs, long min_sources) {
    const int nl = (int)tl.size();
    auto cap_of = [&](int k) { return std::max<long>(min_sources, max_pairs / std::max(1, nt[k])); };
    if (split_long && nl > 0) {  // leaves in parallel: piece counts, offsets, fill
        std::vector<int> p2(nl + 1, 0);
#pragma omp parallel for schedule(static) if (nl >= 4096)
        for (int k = 0; k < nl; ++k) {
            const long cap = cap_of(k);
            long c = 0;
            for (int r = ptr[k]; r < ptr[k + 1]; ++r) c += (rng[2 * r + 1] - rng[2 * r] + cap - 1) / cap;
            p2[k + 1] = (int)c;
        }
        for (int k = 0; k < nl; ++k) p2[k + 1] += p2[k];
        std::vector<int> r2(2 * (size_t)p2[nl]);
#pragma omp parallel for schedule(static) if (nl >= 4096)
        for (int k = 0; k < nl; ++k) {
            const long cap = cap_of(k);
            long q = p2[k];
            for (int r = ptr[k]; r < ptr[k + 1]; ++r)
                for (long b = rng[2 * r]; b < rng[2 * r + 1]; b += cap, ++q) {
                    r2[2 * q] = (int)b;
                    r2[2 * q + 1] = (int)std::min<long>(b + cap, rng[2 * r + 1]);
                }
        }
        ptr.swap(p2);
        rng.swap(r2);
    }
    if (nl == 0) {
        seg.assign(4, 0);
        return false;
    }
    // leaves in parallel: segment counts, offsets, then each leaf fills its own slots
    std::vector<long> soff(nl + 1, 0);
#pragma omp parallel for schedule(static) if (nl >= 4096)
    for (int k = 0; k < nl; ++k) {
        const long cap = cap_of(k);
        long acc = 0, c = 1;
        for (int r = ptr[k]; r < ptr[k + 1]; ++r) {
            const long len = rng[2 * r + 1] - rng[2 * r];
            if (acc > 0 && acc + len > cap) {
                ++c;
                acc = 0;
            }
            acc += len;
        }
        soff[k + 1] = c;
    }
    bool atomic = false;
    for (int k = 0; k < nl; ++k) {
        atomic = atomic || soff[k + 1] > 1;
        soff[k + 1] += soff[k];
    }
    const long nseg = soff[nl];
    std::vector<long> work(nseg);
    std::vector<std::array<int, 4>> body(nseg);
#pragma omp parallel for schedule(static) if (nl >= 4096)
    for (int k = 0; k < nl; ++k) {
        const long cap = cap_of(k), first = soff[k];
        const int multi = soff[k + 1] - first > 1 ? 2 : 0;
        long q = first, acc = 0;
        int r0 = ptr[k];
        auto emit = [&](int r1) {
            work[q] = acc * nt[k];
            body[q] = {tl[k], r0, r1, (q == first ? 1 : 0) | multi};
            ++q;
        };
        for (int r = ptr[k]; r < ptr[k + 1]; ++r) {
            const long len = rng[2 * r + 1] - rng[2 * r];
            if (acc > 0 && acc + len > cap) {
                emit(r);
                r0 = r;
                acc = 0;
            }
            acc += len;
        }
        emit(ptr[k + 1]);
    }
    // descending work, ties in leaf order: a stable LSD radix sort of the segments by
    // (max work - work), 11 bits a pass
    long maxw = 0;
    for (long q = 0; q < nseg; ++q) maxw = std::max(maxw, work[q]);
    std::vector<long> order(nseg), tmp(nseg);
    for (long q = 0; q < nseg; ++q) order[q] = q;
    for (int sh = 0; sh < 63 && (maxw >> sh) > 0; sh += 11) {
        std::array<long, 2049> c{};
        for (long q = 0; q < nseg; ++q) c[1 + (((maxw - work[order[q]]) >> sh) & 2047)]++;
        for (int d = 0; d < 2048; ++d) c[d + 1] += c[d];
        for (long q = 0; q < nseg; ++q) tmp[c[((maxw - work[order[q]]) >> sh) & 2047]++] = order[q];
        order.swap(tmp);
    }
    seg.resize(4 * nseg);
    for (long q = 0; q < nseg; ++q) std::memcpy(&seg[4 * q], body[order[q]].data(), 4 * sizeof(int));
    return atomic;
}

// Work lists of one target set: which nodes need locals, V pairs by operator, X pairs, and
// per target leaf the merged source ranges of its U and W lists.
// Dense index of the V-list operators: (level, source - target lattice offset in [-3, 3]^3).
// M2L operator keys, 5 ints: target level, source level, and the source-minus-target centre offset
// in units of the target node's half-width (per axis).  V pairs (same level, lattice offset o in
// [-3, 3]^3) have offset 2 o and a dense index; X pairs (a coarser source leaf) are hashed.
struct OpIndex {
    std::vector<int> dense;  // level * 343 + offset -> operator id, -1 when absent
    std::vector<int> keys;   // 5 ints per operator
    struct KeyHash {
        size_t operator()(const std::array<int, 5> &k) const {
            uint64_t h = 1469598103934665603ULL;  // FNV-1a over the five ints
            for (int v : k) h = (h ^ (uint32_t)v) * 1099511628211ULL;
            return (size_t)h;
        }
    };
    std::unordered_map<std::array<int, 5>, int, KeyHash> xmap;
    explicit OpIndex(int nlevels) : dense((size_t)std::max(1, nlevels) * 343, -1) {}
    int add(const std::array<int, 5> &k) {
        const int id = (int)keys.size() / 5;
        keys.insert(keys.end(), k.begin(), k.end());
        return id;
    }
    int get(int l, int ox, int oy, int oz) {
        IBIM_REQUIRE(ox >= -3 && ox <= 3 && oy >= -3 && oy <= 3 && oz >= -3 && oz <= 3, "V-list offset out of range");
        int &id = dense[(size_t)l * 343 + (ox + 3) * 49 + (oy + 3) * 7 + (oz + 3)];
        if (id < 0) id = add({l, l, 2 * ox, 2 * oy, 2 * oz});
        return id;
    }
    int get_x(int lt, int ls, int dx, int dy, int dz) {
        const std::array<int, 5> k{lt, ls, dx, dy, dz};
        auto it = xmap.find(k);
        if (it != xmap.end()) return it->second;
        const int id = add(k);
        xmap.emplace(k, id);
        return id;
    }
};

static void build_target_lists(Plan &P, TargetSet &S, OpIndex &opid) {
    const TreeHost &T = P.tree;
    cudaStream_t s = P.ctx->stream;
    const int nn = T.nnodes;
    auto has_t = [&](int i) { return S.end[i] > S.begin[i]; };
    auto has_s = [&](int i) { return T.src_end[i] > T.src_begin[i]; };
    // parents by their children's level; levels 0 and 1 have no locals
    std::vector<int> l2l, lb(T.nlevels + 1, 0);
    for (int l = 0; l < T.nlevels; ++l) {
        lb[l] = (int)l2l.size();
        if (l < 3) continue;
        for (int i = T.level_begin[l - 1]; i < T.level_begin[l]; ++i)
            if (!T.leaf[i] && has_t(i)) l2l.push_back(i);
    }
    lb[T.nlevels] = (int)l2l.size();
    S.l2l_level_begin = lb;
    up_int(S.l2l_parents, l2l, s);
    // V and X pairs grouped by operator with counting sorts: pairs are generated per target node
    // in parallel, new operator keys get ids in key order (V: dense index, X: sorted keys), and
    // each thread scatters its own contiguous node range, so the grouping is deterministic
    std::vector<int> xs, xt;
    std::vector<long> poff(nn + 1, 0);
    std::vector<long> vcount(nn, 0), xcount(nn, 0);
#pragma omp parallel for schedule(static)
    for (int i = 0; i < nn; ++i) {
        if (!has_t(i)) continue;
        long v = 0, x = 0;
        for (int sidx : T.V[i]) v += has_s(sidx);
        for (int sidx : T.X[i]) x += has_s(sidx);
        vcount[i] = v;
        xcount[i] = x;
    }
    for (int i = 0; i < nn; ++i) {
        S.nv_list += vcount[i];
        S.nx_list += xcount[i];
        poff[i + 1] = poff[i] + vcount[i] + (P.x_as_ops ? xcount[i] : 0);
    }
    const long npair = poff[nn];
    HostArr<int> pkey(npair), psrc(npair), ptgt(npair);  // pkey: V dense index, or -1 - X slot
    std::vector<std::array<int, 5>> xkey;
    std::vector<long> xslot_of_pair;
    std::vector<long> xoff(nn + 1, 0);
    if (P.x_as_ops) {
        for (int i = 0; i < nn; ++i) xoff[i + 1] = xoff[i] + xcount[i];
        xkey.resize(xoff[nn]);
    }
    std::vector<int> level_of(nn);
    for (int l = 0; l < T.nlevels; ++l)
        for (int i = T.level_begin[l]; i < T.level_begin[l + 1]; ++i) level_of[i] = l;
    // which dense V keys occur: per-thread flags set while the pairs are generated, OR-ed afterwards
    const size_t nd = opid.dense.size();
    std::vector<std::vector<char>> vused(omp_get_max_threads(), std::vector<char>(nd, 0));
#pragma omp parallel for schedule(dynamic, 64)
    for (int i = 0; i < nn; ++i) {
        if (!has_t(i)) continue;
        const int l = level_of[i];
        char *used_t = vused[omp_get_thread_num()].data();
        long q = poff[i];
        for (int sidx : T.V[i]) {
            if (!has_s(sidx)) continue;
            const int ox = T.coord[3 * sidx] - T.coord[3 * i], oy = T.coord[3 * sidx + 1] - T.coord[3 * i + 1],
                      oz = T.coord[3 * sidx + 2] - T.coord[3 * i + 2];
            pkey[q] = l * 343 + (ox + 3) * 49 + (oy + 3) * 7 + (oz + 3);
            used_t[pkey[q]] = 1;
            psrc[q] = sidx;
            ptgt[q] = i;
            ++q;
        }
        if (!P.x_as_ops) continue;
        long xq = xoff[i];
        for (int sidx : T.X[i]) {
            if (!has_s(sidx)) continue;
            // centre offset in target half-widths: (2 c_s + 1) 2^(lt - ls) - (2 c_t + 1)
            const int ls = level_of[sidx], sh = l - ls;
            std::array<int, 5> k{l, ls, 0, 0, 0};
            for (int a = 0; a < 3; ++a)
                k[2 + a] = (2 * T.coord[3 * sidx + a] + 1) * (1 << sh) - (2 * T.coord[3 * i + a] + 1);
            xkey[xq] = k;
            pkey[q] = -1 - (int)xq;
            psrc[q] = sidx;
            ptgt[q] = i;
            ++q;
            ++xq;
        }
    }
    if (!P.x_as_ops) {
        for (int i = 0; i < nn; ++i) {
            if (!has_t(i)) continue;
            for (int sidx : T.X[i])
                if (has_s(sidx)) {
                    xs.push_back(sidx);
                    xt.push_back(i);
                }
        }
    }
    trace_mark("lists: pairs generated");
    // operator ids: V keys in dense-index order, then X keys in sorted order
    {
        std::vector<char> used(nd, 0);
        for (const auto &part : vused)
            for (size_t d = 0; d < nd; ++d) used[d] |= part[d];
        for (size_t d = 0; d < used.size(); ++d)
            if (used[d]) {
                const int l = (int)(d / 343), c = (int)(d % 343);
                opid.get(l, c / 49 - 3, (c / 7) % 7 - 3, c % 7 - 3);
            }
    }
    std::vector<int> xid(xkey.size());
    const long nx = (long)xkey.size();
    // X keys as 64-bit codes in the same order (levels 5 bits each, offsets 18 bits each biased
    // by 2^17) while every key fits, else the keys themselves: per-thread sorted unique keys,
    // merged; operator ids in sorted key order
    auto fits = [](const std::array<int, 5> &k) {
        return k[0] < 32 && k[1] < 32 && std::abs(k[2]) < (1 << 17) && std::abs(k[3]) < (1 << 17) &&
               std::abs(k[4]) < (1 << 17);
    };
    int all_fit = 1;
#pragma omp parallel for schedule(static) reduction(min : all_fit)
    for (long k = 0; k < nx; ++k) all_fit = std::min(all_fit, fits(xkey[k]) ? 1 : 0);
    auto ids_by_sorted_keys = [&](auto key_of, auto make_op) {
        using K = decltype(key_of(xkey[0]));
        std::vector<K> xc(nx);
        const int nthr = std::max(1, std::min({32, omp_get_max_threads(), (int)(nx / 4096) + 1}));
        std::vector<std::vector<K>> part(nthr);
#pragma omp parallel for schedule(static) num_threads(nthr)
        for (int t = 0; t < nthr; ++t) {
            const long k0 = nx * t / nthr, k1 = nx * (t + 1) / nthr;
            for (long k = k0; k < k1; ++k) xc[k] = key_of(xkey[k]);
            std::vector<K> &u = part[t];
            u.assign(xc.begin() + k0, xc.begin() + k1);
            std::sort(u.begin(), u.end());
            u.erase(std::unique(u.begin(), u.end()), u.end());
        }
        std::vector<K> u;
        for (auto &v : part) u.insert(u.end(), v.begin(), v.end());
        std::sort(u.begin(), u.end());
        u.erase(std::unique(u.begin(), u.end()), u.end());
        std::vector<int> uid(u.size());
        for (size_t k = 0; k < u.size(); ++k) uid[k] = make_op(u[k]);
#pragma omp parallel for schedule(static)
        for (long k = 0; k < nx; ++k) xid[k] = uid[std::lower_bound(u.begin(), u.end(), xc[k]) - u.begin()];
    };
    if (nx > 0 && all_fit) {
        const uint64_t b17 = 1u << 17, m18 = (1u << 18) - 1;
        ids_by_sorted_keys(
            [&](const std::array<int, 5> &k) {
                return ((uint64_t)k[0] << 59) | ((uint64_t)k[1] << 54) | ((uint64_t)(k[2] + b17) << 36) |
                       ((uint64_t)(k[3] + b17) << 18) | (uint64_t)(k[4] + b17);
            },
            [&](uint64_t c) {
                return opid.get_x((int)(c >> 59), (int)((c >> 54) & 31), (int)((c >> 36) & m18) - (int)b17,
                                  (int)((c >> 18) & m18) - (int)b17, (int)(c & m18) - (int)b17);
            });
    } else if (nx > 0) {
        ids_by_sorted_keys([](const std::array<int, 5> &k) { return k; },
                           [&](const std::array<int, 5> &k) { return opid.get_x(k[0], k[1], k[2], k[3], k[4]); });
    }
    trace_mark("lists: operator ids");
    const int nop = (int)opid.keys.size() / 5;
    HostArr<int> pop(npair);
#pragma omp parallel for schedule(static)
    for (long q = 0; q < npair; ++q) pop[q] = pkey[q] >= 0 ? opid.dense[pkey[q]] : xid[-1 - pkey[q]];
    // counting sort by operator; thread t owns pairs [t0, t1) and scatters them in order
    std::vector<long> opbeg(nop + 1, 0);
    HostArr<int> gs(npair), gt(npair);
    {
        const int nthr = std::max(1, std::min({64, omp_get_max_threads(), (int)(npair / 65536) + 1}));
        std::vector<std::vector<long>> hist(nthr, std::vector<long>(nop, 0));
#pragma omp parallel for schedule(static) num_threads(nthr)
        for (int t = 0; t < nthr; ++t) {
            const long t0 = npair * t / nthr, t1 = npair * (t + 1) / nthr;
            for (long q = t0; q < t1; ++q) hist[t][pop[q]]++;
        }
        long run = 0;
        for (int op = 0; op < nop; ++op) {
            opbeg[op] = run;
            for (int t = 0; t < nthr; ++t) {
                const long c = hist[t][op];
                hist[t][op] = run;
                run += c;
            }
        }
        opbeg[nop] = run;
#pragma omp parallel for schedule(static) num_threads(nthr)
        for (int t = 0; t < nthr; ++t) {
            const long t0 = npair * t / nthr, t1 = npair * (t + 1) / nthr;
            for (long q = t0; q < t1; ++q) {
                const long d = hist[t][pop[q]]++;
                gs[d] = psrc[q];
                gt[d] = ptgt[q];
            }
        }
    }
    // chunks (operator, first pair, count) of each contraction's width, in operator order:
    // counts per operator, offsets, then the operators in parallel
    std::vector<int> chunks, chunks32, chunks_tc, chunks_tc2, chunks_oz;
    // `even`: an operator's chunks of like size, multiples of 16, instead of full ones and a rest
    auto cut = [&](std::vector<int> &out, int max_width, bool even = false) {
        auto width_of = [&](int op) {
            const long n = opbeg[op + 1] - opbeg[op], c = (n + max_width - 1) / max_width;
            return even && c > 0 ? std::min<long>(max_width, ((n + c - 1) / c + 15) / 16 * 16) : (long)max_width;
        };
        std::vector<long> coff(nop + 1, 0);
        for (int op = 0; op < nop; ++op) {
            const long w = width_of(op);
            coff[op + 1] = coff[op] + (opbeg[op + 1] - opbeg[op] + w - 1) / w;
        }
        out.resize(3 * coff[nop]);
#pragma omp parallel for schedule(static) if (nop >= 256)
        for (int op = 0; op < nop; ++op) {
            const long b = opbeg[op], n = opbeg[op + 1] - opbeg[op], width = width_of(op);
            long c = coff[op];
            for (long q = 0; q < n; q += width, ++c) {
                out[3 * c] = op;
                out[3 * c + 1] = (int)(b + q);
                out[3 * c + 2] = (int)std::min<long>(width, n - q);
            }
        }
    };
    cut(chunks, M2L_CH);
    cut(chunks32, M2L_CH32);
    cut(chunks_tc, M2L_CHTC);
    cut(chunks_tc2, 2 * M2L_CHTC, true);
    cut(chunks_oz, M2L_CHOZ);
    if (P.oz64_ok) {
        std::vector<int> chunks_oz64;
        cut(chunks_oz64, M2L_CHOZ64);
        S.nchunks_oz64 = (int)chunks_oz64.size() / 3;
        up_int(S.v_chunk_oz64, chunks_oz64, s);
    }
    trace_mark("lists: pairs grouped");
    S.nvpairs = npair;
    S.nchunks = (int)chunks.size() / 3;
    S.nchunks32 = (int)chunks32.size() / 3;
    up_int(S.v_chunk32, chunks32, s);
    S.nchunks_tc = (int)chunks_tc.size() / 3;
    up_int(S.v_chunk_tc, chunks_tc, s);
    S.nchunks_tc2 = (int)chunks_tc2.size() / 3;
    up_int(S.v_chunk_tc2, chunks_tc2, s);
    S.nchunks_oz = (int)chunks_oz.size() / 3;
    up_int(S.v_chunk_oz, chunks_oz, s);
    S.v_src.alloc(std::max<long>(1, npair), s);
    S.v_src.upload(gs.data(), npair);
    S.v_tgt.alloc(std::max<long>(1, npair), s);
    S.v_tgt.upload(gt.data(), npair);
    up_int(S.v_chunk, chunks, s);
    S.nxpairs = (long)xs.size();
    up_int(S.x_src, xs, s);
    up_int(S.x_tgt, xt, s);
    trace_mark("lists: chunks, uploads");
    // target leaves and the near-field pair count (U and W lists); the FP64 kernel's merged
    // source ranges are built on first use (near64_lists)
    std::vector<int> tl;
    for (int i = 0; i < nn; ++i)
        if (T.leaf[i] && has_t(i)) tl.push_back(i);
    long npairs = 0;
#pragma omp parallel for schedule(dynamic, 64) reduction(+ : npairs)
    for (long k = 0; k < (long)tl.size(); ++k) {
        const int i = tl[k];
        long nsrc = 0;
        for (int sidx : T.U[i]) nsrc += T.src_end[sidx] - T.src_begin[sidx];
        for (int sidx : T.W[i]) nsrc += T.src_end[sidx] - T.src_begin[sidx];
        npairs += nsrc * (S.end[i] - S.begin[i]);
    }
    S.ntleaves = (int)tl.size();
    S.near_pairs = npairs;
    S.tl_h = tl;
    up_int(S.tleaf, tl, s);
    up_int(S.tbeg, S.begin, s);
    up_int(S.tend, S.end, s);
    S.out4.alloc((size_t)4 * std::max<long>(1, S.nt), s);
}

// Extra targets (e.g. atom centres): descend the source tree with the split rule of
// assignChildren (bbfmm.cpp:121-131) and keep each node's targets contiguous in DFS order.
static void bin_targets(Plan &P, TargetSet &S, const double *pts, long nt, const std::vector<int> &child_first) {
    const TreeHost &T = P.tree;
    const int nn = T.nnodes;
    std::vector<int> dfs(nn, 0);
    {
        std::vector<int> stack{0};
        int k = 0;
        while (!stack.empty()) {
            const int n = stack.back();
            stack.pop_back();
            dfs[n] = k++;
            if (!T.leaf[n])
                for (int c = 7; c >= 0; --c) stack.push_back(child_first[n] + c);
        }
    }
    std::vector<int> leaf_of(nt);
    for (long i = 0; i < nt; ++i) {
        const double *x = pts + 3 * i;
        int n = 0;
        while (!T.leaf[n]) {
            const double *c = &T.center[3 * n];
            const int ch = 4 * (x[2] < c[2] ? 0 : 1) + 2 * (x[1] < c[1] ? 0 : 1) + (x[0] < c[0] ? 0 : 1);
            n = child_first[n] + ch;
        }
        leaf_of[i] = n;
    }
    S.perm.resize(nt);
    for (long i = 0; i < nt; ++i) S.perm[i] = (int)i;
    std::stable_sort(S.perm.begin(), S.perm.end(), [&](int a, int b) { return dfs[leaf_of[a]] < dfs[leaf_of[b]]; });
    S.begin.assign(nn, 0);
    S.end.assign(nn, 0);
    std::vector<int> cnt(nn, 0);
    for (long i = 0; i < nt; ++i) cnt[leaf_of[i]]++;
    // leaves in DFS order get consecutive ranges; internal nodes span their children
    std::vector<int> order(nn);
    for (int i = 0; i < nn; ++i) order[dfs[i]] = i;
    int off = 0;
    for (int q = 0; q < nn; ++q) {
        const int n = order[q];
        if (T.leaf[n]) {
            S.begin[n] = off;
            S.end[n] = off + cnt[n];
            off += cnt[n];
        }
    }
    for (int n = nn - 1; n >= 0; --n)
        if (!T.leaf[n]) {
            S.begin[n] = S.begin[child_first[n]];
            S.end[n] = S.end[child_first[n] + 7];
        }
}

Plan *make_plan(Tube *t, bool with_self, const double *extra, long n_extra, int order, int maxpoint, int maxlevel,
                int precision) {
    IBIM_REQUIRE(order >= 2 && order <= MAXP, "fmm_np must be in [2, 8]");
    IBIM_REQUIRE(precision == IBIM_PRECISION_FP64 || precision == IBIM_PRECISION_MIXED ||
                     precision == IBIM_PRECISION_FP64_TC,
                 "unknown precision");
    IBIM_REQUIRE(t && t->n > 0, "plan needs a non-empty tube");
    IBIM_REQUIRE(with_self || (extra && n_extra > 0), "plan needs targets");
    Ctx *c = t->ctx;
    cudaStream_t s = c->stream;
    const long ns = t->n;
    std::vector<double> pts(3 * ns);
    {
        // through the context's pinned staging buffer
        double *h = static_cast<double *>(c->pinned_buffer(sizeof(double) * 3 * (size_t)ns));
        t->x.download(h, ns);
        t->y.download(h + ns, ns);
        t->z.download(h + 2 * ns, ns);
        IBIM_CUDA(cudaStreamSynchronize(s));
#pragma omp parallel for schedule(static) if (ns >= (1 << 16))
        for (long i = 0; i < ns; ++i) {
            pts[3 * i] = h[i];
            pts[3 * i + 1] = h[ns + i];
            pts[3 * i + 2] = h[2 * ns + i];
        }
    }
    Plan *P = new Plan();
    P->ctx = c;
    P->tube = t;
    // X pairs join the operator contraction; IBIM_X_ONTHEFLY keeps the on-the-fly X kernels
    // (kernel evaluated per pair, no operator storage)
    P->x_as_ops = std::getenv("IBIM_X_ONTHEFLY") == nullptr;
    P->ns = ns;
    P->p = order;
    P->R = order * order * order;
    P->maxpoint = maxpoint;
    P->maxlevel = maxlevel;
    P->precision = precision;
    P->tune = tuning_for(order, ns);
    P->oz64_ok = precision == IBIM_PRECISION_FP64 && m2l_oz64_fits(order, 0.);
    try {
        trace_mark("plan: coordinates downloaded");
        P->tree = build_tree(pts.data(), ns, pts.data(), ns, maxpoint, maxlevel);
        trace_mark("plan: tree and lists");
        TreeHost &T = P->tree;
        const int nn = T.nnodes, R = P->R, n4 = 4 * R;
        T.p = order;
        T.R = R;
        P->src_perm.alloc(ns, s);
        P->src_perm.upload(T.src_perm.data(), ns);
        DevBuf<double> *dst[7] = {&P->sx, &P->sy, &P->sz, &P->snx, &P->sny, &P->snz, &P->sw};
        const DevBuf<double> *srcs[7] = {&t->x, &t->y, &t->z, &t->nx, &t->ny, &t->nz, &t->w};
        const double h3 = t->h * t->h * t->h;
        for (int k = 0; k < 7; ++k) {
            dst[k]->alloc(ns, s);
            // quadrature weight = w * s * h^3 with s = 1 (electric.cpp:33)
            plan_gather(c, ns, P->src_perm.ptr, srcs[k]->ptr, dst[k]->ptr, k == 6 ? h3 : 1.0);
        }
        P->ncenter.alloc(3 * nn, s);
        P->ncenter.upload(T.center.data(), 3 * nn);
        P->nradius.alloc(3 * nn, s);
        P->nradius.upload(T.radius.data(), 3 * nn);
        up_int(P->nsrc_begin, T.src_begin, s);
        up_int(P->nsrc_end, T.src_end, s);
        up_int(P->nparent, T.parent, s);
        up_int(P->nempty, T.empty, s);
        std::vector<int> child_first(nn, -1);
        for (int i = nn - 1; i >= 0; --i)
            if (T.parent[i] >= 0) child_first[T.parent[i]] = i - T.index8[i];
        up_int(P->nchild_first, child_first, s);
        auto has_s = [&](int i) { return T.src_end[i] > T.src_begin[i]; };
        std::vector<int> p2m, need(nn, 0);
        for (int i = 0; i < nn; ++i)
            if (T.leaf[i] && has_s(i)) p2m.push_back(i);
        // no list holds a multipole of levels 0 and 1 but a leaf's own: the upward pass ends at level 2
        for (int l = 3; l < T.nlevels; ++l)
            for (int i = T.level_begin[l]; i < T.level_begin[l + 1]; i += 8) {
                int k = 0;
                for (int c = 0; c < 8; ++c) k += has_s(i + c);
                for (int c = 0; c < 8; ++c) need[i + c] = k;
            }
        up_int(P->p2m_nodes, p2m, s);
        up_int(P->up_need, need, s);
        P->up_count.alloc(nn, s);
        P->up_count.zero();
        P->np2m = (int)p2m.size();
        OpIndex opid(T.nlevels);
        trace_mark("plan: node arrays enqueued");
        if (with_self) {
            TargetSet *S = new TargetSet();
            P->targets.push_back(S);
            S->self = true;
            S->nt = ns;
            S->begin = T.src_begin;
            S->end = T.src_end;
            S->perm = T.src_perm;
            up_int(S->perm_d, S->perm, s);
            build_target_lists(*P, *S, opid);
            trace_mark("plan: self target lists");
        }
        if (extra && n_extra > 0) {
            TargetSet *S = new TargetSet();
            P->targets.push_back(S);
            S->nt = n_extra;
            bin_targets(*P, *S, extra, n_extra, child_first);
            std::vector<double> tq[3];
            for (int a = 0; a < 3; ++a) {
                tq[a].resize(n_extra);
                for (long i = 0; i < n_extra; ++i) tq[a][i] = extra[3 * (long)S->perm[i] + a];
            }
            S->tx.alloc(n_extra, s);
            S->ty.alloc(n_extra, s);
            S->tz.alloc(n_extra, s);
            S->tx.upload(tq[0].data(), n_extra);
            S->ty.upload(tq[1].data(), n_extra);
            S->tz.upload(tq[2].data(), n_extra);
            up_int(S->perm_d, S->perm, s);
            build_target_lists(*P, *S, opid);
            trace_mark("plan: extra target lists");
        }
        P->nops = (int)opid.keys.size() / 5;
        P->oz64_ok = P->oz64_ok && m2l_oz64_fits(order, P->nops);
        P->op_key_h = opid.keys;
        if (P->op_key_h.empty()) P->op_key_h.assign(5, 0);
        up_int(P->op_key, P->op_key_h, s);
        // classes of mirror images: equal levels, offsets equal but for signs
        std::vector<int> ord(P->nops);
        for (int i = 0; i < P->nops; ++i) ord[i] = i;
        const int *key = P->op_key_h.data();
        auto cmp = [&](int a, int b) {
            for (int q = 0; q < 5; ++q) {
                const int u = std::abs(key[5 * a + q]), v = std::abs(key[5 * b + q]);
                if (u != v) return u < v ? -1 : 1;
            }
            return 0;
        };
        std::sort(ord.begin(), ord.end(), [&](int a, int b) {
            const int c = cmp(a, b);
            return c != 0 ? c < 0 : a < b;
        });
        P->op_cls_h.assign(1, 0);
        for (int i = 1; i <= P->nops; ++i)
            if (i == P->nops || cmp(ord[i - 1], ord[i]) != 0) P->op_cls_h.push_back(i);
        up_int(P->op_ord, ord, s);
        up_int(P->op_cls, P->op_cls_h, s);
        ChebTables ht;
        cheb_tables_host(order, ht);
        P->tables.alloc(1, s);
        P->tables.upload(&ht, 1);
        P->root_r.alloc(3, s);
        P->root_r.upload(T.radius.data(), 3);
        P->mult.alloc((size_t)nn * n4, s);
        P->local.alloc((size_t)nn * n4, s);
        P->dens4.alloc((size_t)4 * ns, s);
        static std::atomic<uint64_t> split, split_near;
        near64_side_by_side(split_near);
        side_by_side(split, {(const void *)k_gather});
        const size_t sm = sizeof(double) * M2L_CH * n4;
        if (sm > 48 * 1024)
            IBIM_CUDA(cudaFuncSetAttribute(k_m2l_v64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        IBIM_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        delete P;
        throw;
    }
    return P;
}

void fmm_prepare_operators(Plan &P, const ibim_kernel_params &kp, int precision) {
    const double key[5] = {kp.kappa, kp.dE, kp.dI, kp.tau, (double)kp.k3_scaled};
    const bool is64 = precision == IBIM_PRECISION_FP64;
    double *cache = is64 ? P.kp64 : P.kp32;
    bool same = is64 ? P.ops64_ready : P.ops32_ready;
    for (int i = 0; i < 5; ++i) same = same && cache[i] == key[i];
    if (same || P.nops == 0) return;
    cudaStream_t s = P.ctx->stream;
    const int R = P.R, n4 = 4 * R;
    const KParams k = make_kparams(kp, P.tube->h);
    if (precision == IBIM_PRECISION_FP64) {
        P.ops64.alloc((size_t)P.nops * n4 * n4, s);
        dim3 g(div_up((long)R * R, 256), (int)P.op_cls_h.size() - 1);
        { ProfScope ps_(PROF_OPS); (count_launch(), k_make_ops64<<<g, 256, 0, s>>>(P.tables.ptr, P.op_key.ptr, P.root_r.ptr, k, ENTRY_BLOCK, P.op_cls.ptr, P.op_ord.ptr, -1, P.ops64.ptr)); }
        IBIM_CHECK_LAUNCH();
    } else {
        bool have64 = P.ops64_ready;
        for (int i = 0; i < 5; ++i) have64 = have64 && P.kp64[i] == key[i];
        fmm_prepare_operators_mixed(P, k, have64 ? P.ops64.ptr : nullptr);
    }
    for (int i = 0; i < 5; ++i) cache[i] = key[i];
    (is64 ? P.ops64_ready : P.ops32_ready) = true;
}

static void kp_key(const ibim_kernel_params &kp, double key[5]) {
    key[0] = kp.kappa;
    key[1] = kp.dE;
    key[2] = kp.dI;
    key[3] = kp.tau;
    key[4] = (double)kp.k3_scaled;
}

static bool same_key(const double a[5], const double b[5]) {
    for (int i = 0; i < 5; ++i)
        if (a[i] != b[i]) return false;
    return true;
}

void fmm_ensure_tc_images(Plan &P, const ibim_kernel_params &kp) {
    double key[5];
    kp_key(kp, key);
    if (P.tc_ready && same_key(P.tc_key, key)) return;
    if (m2l_tc_fp16_form() && P.opsff_ready && same_key(P.kpff, key)) {
        m2l_tc_pack(P, P.opsff.ptr);  // FP16 images from the float-float operators of the digit images
    } else {
        fmm_prepare_operators(P, kp, IBIM_PRECISION_MIXED);
        m2l_tc_pack(P);
    }
    // the images replace the FP32 operators on this path
    P.ops32.release();
    P.ops32_ready = false;
    for (int i = 0; i < 5; ++i) P.tc_key[i] = key[i];
    P.tc_ready = true;
}

void fmm_ensure_oz_images(Plan &P, const ibim_kernel_params &kp) {
    double key[5];
    kp_key(kp, key);
    if (P.oz_ready && same_key(P.oz_key, key)) return;
    if (P.precision != IBIM_PRECISION_FP64 && ops_ff_enabled()) {
        // FP64-class plans: operators in float-float on the FP32 pipes (2^-44 a value, below the
        // digit cut's 2^-43)
        fmm_prepare_operators_ff(P, kp);
        m2l_oz_pack(P, P.opsff.ptr);
    } else {
        fmm_prepare_operators(P, kp, IBIM_PRECISION_FP64);
        m2l_oz_pack(P);
    }
    for (int i = 0; i < 5; ++i) P.oz_key[i] = key[i];
    P.oz_ready = true;
}

bool fmm_ensure_images_ff(Plan &P, const ibim_kernel_params &kp) {
    if (P.precision == IBIM_PRECISION_FP64 || !ops_ff_enabled() || !m2l_tc_fp16_form()) return false;
    double key[5];
    kp_key(kp, key);
    if (P.oz_ready && same_key(P.oz_key, key) && P.tc_ready && same_key(P.tc_key, key)) return true;
    fmm_prepare_operators_ff(P, kp);
    m2l_pack_images_ff(P, P.opsff.ptr);
    const char *chk = std::getenv("IBIM_CHECK_IMAGES");  // read per call: a test switch
    if (chk && chk[0] == '1') m2l_check_images_ff(P, P.opsff.ptr);
    // the images replace the FP32 operators on this path
    P.ops32.release();
    P.ops32_ready = false;
    for (int i = 0; i < 5; ++i) P.oz_key[i] = P.tc_key[i] = key[i];
    P.oz_ready = P.tc_ready = true;
    return true;
}

void fmm_release_fp64_operators(Plan &P) {
    P.ops64.release();
    P.ops64_ready = false;
    P.opsff.release();
    P.opsff_ready = false;
}

// Merged U and W source ranges per target leaf and their work segments, for the FP64 near-field
// kernel (leaves in parallel, concatenated in leaf order).
void near64_lists(Plan &P, TargetSet &S) {
    if (S.near64_ready) return;
    const TreeHost &T = P.tree;
    cudaStream_t s = P.ctx->stream;
    const std::vector<int> &tl = S.tl_h;
    std::vector<std::vector<int>> per(tl.size());
#pragma omp parallel for schedule(dynamic, 32)
    for (long k = 0; k < (long)tl.size(); ++k) {
        const int i = tl[k];
        std::vector<std::pair<int, int>> rg;
        for (int sidx : T.U[i])
            if (T.src_end[sidx] > T.src_begin[sidx]) rg.push_back({T.src_begin[sidx], T.src_end[sidx]});
        for (int sidx : T.W[i])
            if (T.src_end[sidx] > T.src_begin[sidx]) rg.push_back({T.src_begin[sidx], T.src_end[sidx]});
        std::sort(rg.begin(), rg.end());
        std::vector<int> &mg = per[k];
        for (auto &r : rg) {
            if (!mg.empty() && mg.back() == r.first)
                mg.back() = r.second;
            else {
                mg.push_back(r.first);
                mg.push_back(r.second);
            }
        }
    }
    std::vector<int> nptr{0}, nr;
    for (size_t k = 0; k < tl.size(); ++k) {
        nr.insert(nr.end(), per[k].begin(), per[k].end());
        nptr.push_back((int)nr.size() / 2);
    }
    std::vector<int> ntk(tl.size()), seg;
    for (size_t k = 0; k < tl.size(); ++k) ntk[k] = (int)(S.end[tl[k]] - S.begin[tl[k]]);
    // at least eight segments a CTA of the launch (2^11 to 2^14 pairs): with 2^17 the last segments
    // ran alone for most of a small plan's launch (60 atoms: 195 segments, 9.5 ms for 2.6e7 pairs)
    const long cap = std::min(1L << 14, std::max(1L << 11, S.near_pairs / (8L * NEAR_CPS * P.ctx->num_sms)));
    S.near_atomic = near_segments(tl, ntk, nptr, nr, true, seg, cap, 32);
    S.nnear_seg = tl.empty() ? 0 : (int)seg.size() / 4;
    up_int(S.near_seg, seg, s);
    up_int(S.near_ptr, nptr, s);
    up_int(S.near_range, nr, s);
    S.near64_ready = true;
}

// The FP64 operator's digit images, whole or of one entry of the block: the operators in blocks of at most
// 1 GB, each cut and dropped.
static void build_oz64_images(Plan &P, const KParams &k, int entry) {
    cudaStream_t s = P.ctx->stream;
    const int R = P.R, n = entry == ENTRY_BLOCK ? 4 * R : R;
    const size_t per = (size_t)n * n;
    const std::vector<int> &cls = P.op_cls_h;
    const int ncls = (int)cls.size() - 1;
    const int block = (int)std::min<size_t>(std::max(1, P.nops), std::max<size_t>(8, (1UL << 30) / (8 * per)));
    m2l_oz64_alloc(P, entry, k);
    DevBuf<double> ops;
    ops.alloc(per * block, s);
    ProfScope ps_(PROF_OPS);
    for (int c = 0, e; c < ncls; c = e) {  // classes are blockIdx.y
        for (e = c; e < ncls && e - c < 65535 && cls[e + 1] - cls[c] <= block;) ++e;
        (count_launch(), k_make_ops64<<<dim3(div_up((long)R * R, 256), e - c), 256, 0, s>>>(
            P.tables.ptr, P.op_key.ptr, P.root_r.ptr, k, entry, P.op_cls.ptr + c, P.op_ord.ptr, cls[c], ops.ptr));
        IBIM_CHECK_LAUNCH();
        m2l_oz64_pack(P, entry, ops.ptr, P.op_ord.ptr + cls[c], cls[e] - cls[c]);
    }
}

// The images take about twice the memory of the operators that k_m2l_v64 reads, so a plan whose neighbours leave the
// device too little for them takes that contraction (a single kernel: the block), for the rest of its life, instead of
// failing.  Images of single kernels, which the plan keeps between calls, go first.
bool fmm_ensure_oz64_images(Plan &P, const ibim_kernel_params &kp, int entry) {
    if (!P.oz64_ok) return false;
    double key[5];
    kp_key(kp, key);
    auto &Z = P.oz64[entry];
    if (Z.ready && same_key(Z.key, key)) return true;
    Z.ready = false;
    const KParams k = make_kparams(kp, P.tube->h);
    auto drop = [](Plan::Oz64 &z) {
        z.ready = false;
        z.a.release();
        z.sig.release();
    };
    for (int attempt = 0; attempt < 2; ++attempt) {
        try {
            if (Z.a.ptr || m2l_oz64_room(P, entry)) {
                build_oz64_images(P, k, entry);
                for (int i = 0; i < 5; ++i) Z.key[i] = key[i];
                Z.ready = true;
                return true;
            }
        } catch (const Error &e) {
            if (e.status != IBIM_ERR_OUT_OF_MEMORY) throw;
        }
        drop(Z);
        for (int i = 0; i < ENTRY_BLOCK; ++i) drop(P.oz64[i]);
    }
    if (entry == ENTRY_BLOCK) {
        P.oz64_ok = false;
        P.oz64_b.release();
        P.oz64_tau.release();
    }
    return false;
}

void fmm_prepare_fp64(Plan &P, const ibim_kernel_params &kp) {
    if (!fmm_ensure_oz64_images(P, kp, ENTRY_BLOCK)) fmm_prepare_operators(P, kp, IBIM_PRECISION_FP64);
}

// A scalar kernel's FMM as its entry of the block: one component a node, R x R operators instead of 4R x 4R
// (a sixteenth of the products, images of their own built on the first call of each kernel and kept), half
// the near field's instructions.  150 atoms at order 6: 16.5 -> 3.3 ms a product, 40 -> 18 ms the first one.
// Plans without room for all 16 entries' images beside the block's, without digit images, or with X pairs
// evaluated on the fly run the block with the other densities zero.  Builds the entry's images.
bool fmm_one_entry(Plan &P, const ibim_kernel_params &kp, int entry) {
    return P.precision == IBIM_PRECISION_FP64 && P.oz64_ok && P.x_as_ops && m2l_oz64_fits(P.p, P.nops, true) &&
           fmm_ensure_oz64_images(P, kp, entry);
}

// One FP64 FMM: dens (nc x ns, tree order) -> out (nc x nt of target set ts, tree order), nc = 4 for the block,
// 1 for one entry of it.  m2l_sliced: the V-list M2L by exact BF16 slices and the near field in float-float (FP64-class
// accuracy), the mixed path's refinement residual.
static void fmm_run_fp64(Plan &P, int ts, const ibim_kernel_params &kpp, const double *dens, double *out, bool m2l_sliced,
                         int entry = ENTRY_BLOCK) {
    IBIM_REQUIRE(ts >= 0 && ts < (int)P.targets.size(), "no such target set");
    const bool use_oz = m2l_sliced && (4 * P.R + 15) / 16 * 16 <= M2L_OZ_MAXK;
    const bool use_oz64 = !m2l_sliced && fmm_ensure_oz64_images(P, kpp, entry);
    IBIM_REQUIRE(use_oz64 || entry == ENTRY_BLOCK, "the plan has no images of single kernels");
    if (use_oz)
        fmm_ensure_oz_images(P, kpp);
    else if (!use_oz64)
        fmm_prepare_operators(P, kpp, IBIM_PRECISION_FP64);
    const TargetSet &S = *P.targets[ts];
    Ctx *c = P.ctx;
    cudaStream_t s = c->stream;
    const int nc = entry == ENTRY_BLOCK ? 4 : 1;
    const int R = P.R, n4 = nc * R;
    const KParams kp = make_kparams(kpp, P.tube->h);
    const double *tx = S.self ? P.sx.ptr : S.tx.ptr;
    const double *ty = S.self ? P.sy.ptr : S.ty.ptr;
    const double *tz = S.self ? P.sz.ptr : S.tz.ptr;
    // near field (U and W lists, bbfmm.h:571-609): depends only on the densities.  With the
    // overlap on it starts on the auxiliary stream at full occupancy, CTAs taking work segments
    // from a counter, beside the far field; the L2P follows the join (see fmm_run_mixed).  The
    // FP64-class path evaluates it in float-float on the FP32 pipes over the FP32 near lists.
    const bool ff = m2l_sliced && near_ff_enabled() && S.ntleaves > 0;
    KParamsFF kff{};
    if (ff) {
        prepare_mixed(P, *P.targets[ts]);
        kff = make_kparams_ff(kp);
        near_ff_pack(P, dens, s);
    }
    if (!ff && S.ntleaves > 0) near64_lists(P, *P.targets[ts]);
    const int nseg = ff ? S.nnearff_seg : S.nnear_seg;
    const bool atomic = ff ? S.nearff_atomic : S.near_atomic;
    auto near = [&](cudaStream_t st, int l2p_mask, int grid, int *next, bool count_work) {
        if (ff) {
            ProfScope ps_(PROF_NEARFF, count_work ? NEAR_FF_FLOPS * S.near_pairs : 0.,
                          count_work ? 64.0 * P.ns + 40.0 * S.nt : 0., st);
            near_ff_run(P, S, kff, out, st, grid, next);
            return;
        }
        ProfScope ps_(PROF_NEAR64, count_work ? 70.0 * S.near_pairs : 0., count_work ? 56.0 * P.ns + 40.0 * S.nt : 0.,
                      st);
        const Near64K nk = make_near64(kp);
        // the fast forms take FP32 seeds of d2 >= (tau h)^2 and n >= 0 of 2^(-n / 512)
        const int mode = !(kp.vr2 >= 1e-30) ? NEAR_GENERAL
                                            : (kp.kappa > 0. ? NEAR_YUKAWA : (kp.kappa == 0. ? NEAR_LAPLACE : NEAR_GENERAL));
        const int slot = entry & 3, field = entry >> 2;
        const int kind = entry == ENTRY_BLOCK ? NEAR_BLOCK
                         : field == 0         ? (slot == 3 ? NEAR_K2 : NEAR_K1)
                                              : (slot == 3 ? NEAR_K4 : NEAR_K3);
        auto kern = near64_kernel(mode, kind);
        (count_launch(), kern<<<grid, NEAR_T, 0, st>>>(P.tables.ptr, P.exp_tab.ptr, nk, reinterpret_cast<const int4 *>(S.near_seg.ptr),
                                                       S.near_range.ptr, S.tbeg.ptr, S.tend.ptr, P.ncenter.ptr,
                                                       P.nradius.ptr, P.sx.ptr, P.sy.ptr, P.sz.ptr, dens, P.ns, tx, ty,
                                                       tz, S.nt, P.local.ptr, out, l2p_mask, S.nnear_seg, next, slot,
                                                       field - 1));
    };
    const bool overlap = near_overlap() && S.ntleaves > 0;
    if (!P.exp_tab.ptr) {
        std::vector<double> h(NEAR_EXP);
        for (int j = 0; j < NEAR_EXP; ++j) h[j] = std::exp2(-(double)j / NEAR_EXP);
        P.exp_tab.alloc(NEAR_EXP, s);
        P.exp_tab.upload(h.data(), NEAR_EXP);
        IBIM_CUDA(cudaStreamSynchronize(s));
    }
    const int full = (ff ? near_ff_occupancy() : NEAR_CPS) * c->num_sms;
    // Beside the FP64 operator's digit products the near field starts when they do, not with the P2M: the upward
    // pass has the FP64 pipe to itself (2,000 atoms: 61.9 -> 56.9 ms a matvec).  It has to be resident
    // before the products' CTAs queue, which a lower priority would wait for: m2l_oz64_run calls fork
    // ahead of its split kernel.
    // So does the float-float one beside the residual's products, with two CTAs an SM (what their shared memory
    // leaves) and a drain launch (2,000-atom solve: 86.4 ms of GMRES with the near field first, 85.1 and 84.8
    // with one and two); merged plans, whose chunks stop molecule by molecule, gain nothing and keep it first.
    const bool with_m2l = use_oz64 ? S.nchunks_oz64 > 0 : ff && use_oz && !P.batched && S.nchunks_oz > 0;
    const int side = near_side_ctas() > 0 ? near_side_ctas() * c->num_sms
                                          : std::min(full, ff && with_m2l ? 2 * c->num_sms : full);
    bool forked = false;
    auto fork = [&] {
        IBIM_CUDA(cudaEventRecord(c->ev_near_fork, s));
        IBIM_CUDA(cudaStreamWaitEvent(c->aux, c->ev_near_fork, 0));
        near(c->aux, 0, std::min(nseg, side), P.near_next.ptr, true);
        IBIM_CUDA(cudaEventRecord(c->ev_near_join, c->aux));
        forked = true;
    };
    const std::function<void()> beside = overlap && with_m2l ? std::function<void()>(fork) : nullptr;
    if (overlap) {
        if (!P.near_next.ptr) P.near_next.alloc(1, s);
        IBIM_CUDA(cudaMemsetAsync(P.near_next.ptr, 0, sizeof(int), s));
        if (atomic) IBIM_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * nc * S.nt, s));
        if (!with_m2l) fork();
    }
    try {
        translate_up(P, nc, dens, P.mult.ptr);
        P.local.zero();
        if (use_oz) {
            m2l_oz_run(P, S, beside);
        } else if (use_oz64) {
            m2l_oz64_run(P, S, entry, beside);
        } else if (S.nchunks > 0) {
            ProfScope ps_(PROF_M2L_V64, 2.0 * n4 * (double)n4 * S.nvpairs,
                          8.0 * n4 * (2.0 * S.nvpairs + (double)n4 * P.nops));
            (count_launch(), k_m2l_v64<<<S.nchunks, 256, sizeof(double) * M2L_CH * n4, s>>>(
                 n4, S.v_chunk.ptr, S.v_src.ptr, S.v_tgt.ptr, P.ops64.ptr, P.mult.ptr, P.local.ptr));
        }
        if (S.nxpairs > 0) {
            ProfScope ps_(PROF_M2L_X64, 102.0 * R * (double)R * S.nxpairs, 16.0 * n4 * S.nxpairs);
            (count_launch(), k_m2l_x64<<<(int)S.nxpairs, 128, 0, s>>>(P.tables.ptr, kp, S.x_src.ptr, S.x_tgt.ptr,
                                                                      P.ncenter.ptr, P.nradius.ptr, P.mult.ptr,
                                                                      P.local.ptr));
        }
        translate_down(P, S, nc, P.local.ptr);
    } catch (...) {
        if (forked) cudaStreamSynchronize(c->aux);  // the near field still reads dens and writes out
        throw;
    }
    if (S.ntleaves > 0) {
        if (overlap) {
            if (side < std::min(nseg, full)) near(s, 0, std::min(nseg, full), P.near_next.ptr, false);
            IBIM_CUDA(cudaStreamWaitEvent(s, c->ev_near_join, 0));
        } else {
            if (atomic) IBIM_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * nc * S.nt, s));
            near(s, 1, nseg, nullptr, true);
        }
        // the L2P runs on its own after the near field
        if (overlap || ff) translate_l2p(P, S, nc, tx, ty, tz, P.local.ptr, out);
    }
    IBIM_CHECK_LAUNCH();
}

void fmm_run_entry(Plan &P, int ts, const ibim_kernel_params &kp, const double *dens, double *out, int entry) {
    fmm_run_fp64(P, ts, kp, dens, out, false, entry);
}

void fmm_run(Plan &P, int ts, const ibim_kernel_params &kp, const double *dens, double *out, int precision) {
    if (precision == IBIM_PRECISION_FP64)
        fmm_run_fp64(P, ts, kp, dens, out, false);
    else if (precision == IBIM_PRECISION_FP64_TC)
        fmm_run_fp64(P, ts, kp, dens, out, m2l_tc_supported());
    else
        fmm_run_mixed(P, ts, kp, dens, out);
}

}  // namespace ibim
