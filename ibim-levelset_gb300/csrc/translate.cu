// Chebyshev translations of the FMM: sources up to multipoles (bbfmm.h:507-534), locals down to targets
// (bbfmm.h:566-567, :600), in FP64 and FP32, with nc = 4 components a node (the fused operator) or 1.
//
// All are small tensor contractions along one axis at a time.  Compiled per order: a thread owns one line of p
// nodes in registers, so an entry of the transfer matrix serves p outputs, and no index is divided at run time.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "fmm_common.cuh"

namespace ibim {

namespace {

template <class T, int P, int NC> struct Shape {
    static constexpr int R = P * P * P, N = NC * R;
    static constexpr int NL = NC * P * P;                               // lines of P nodes
    static constexpr int UP_T = NL <= 128 ? 128 : (NL + 31) / 32 * 32;  // threads of the upward kernel
    static constexpr int G = UP_T / NL;                                 // groups of lines that share the P2M's points
    static constexpr int V = 16 / sizeof(T), PX = (P + V - 1) / V * V;  // rows read by 16-byte loads
    static constexpr int UP_SMEM = 6 * N * (int)sizeof(T);
    static constexpr int P2M_SMEM = 32 * (PX + 2 * P + NC) * (int)sizeof(T), RED_SMEM = G * N * (int)sizeof(T);
    static constexpr int SMEM = std::max({UP_SMEM, P2M_SMEM, RED_SMEM});
    static constexpr int L2P_W = 4;                                     // leaves (warps) a CTA of the L2P
};

template <class T, int P, int PX> struct alignas(16) Row { T v[PX]; };

// Tables of order P in shared memory: the transfer matrices as rows over the parent's nodes (S) or the child's (St).
template <class T, int P, int PX, bool DOWN>
__device__ __forceinline__ void load_transfer(Row<T, P, PX> (*S)[P], const ChebTables *__restrict__ tab) {
    for (int i = threadIdx.x; i < 2 * P * P; i += blockDim.x) {
        const int b = i / (P * P), k = i / P % P, n = i % P;
        if (DOWN) S[b][n].v[k] = (T)tab->S[b][k][n];
        else S[b][k].v[n] = (T)tab->S[b][k][n];
    }
}

template <class T, int P> struct Interp {
    T node[P][P];  // T_k(cheb_m): [m][k]
    __device__ __forceinline__ void load(const ChebTables *__restrict__ tab) {
        for (int i = threadIdx.x; i < P * P; i += blockDim.x) node[i / P][i % P] = (T)tab->tnode[i / P][i % P];
    }
    // S_p(x, cheb_m), m < p: (-1 + 2 sum_k T_k(x) T_k(cheb_m)) / p (bbfmm.h:409-419)
    template <class O> __device__ __forceinline__ void at(T x, O out) const {
        T t[P];
        t[0] = T(1);
        if (P > 1) t[1] = x;
#pragma unroll
        for (int k = 2; k < P; ++k) t[k] = T(2) * x * t[k - 1] - t[k - 2];
#pragma unroll
        for (int m = 0; m < P; ++m) {
            T s = T(0);
#pragma unroll
            for (int k = 0; k < P; ++k) s = fma(t[k], node[m][k], s);
            out(m, (T(-1) + T(2) * s) * (T(1) / T(P)));
        }
    }
};

// out[i] += sum_k in[k] S[k][i]
template <class T, int P, int PX>
__device__ __forceinline__ void line(const T (&in)[P], const Row<T, P, PX> *S, T (&out)[P]) {
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const Row<T, P, PX> s = S[k];
#pragma unroll
        for (int n = 0; n < P; ++n) out[n] = fma(in[k], s.v[n], out[n]);
    }
}

// Coordinate of a point in its leaf's box, in half-widths: FP64 from absolute coordinates, FP32 from
// leaf-relative ones.
__device__ __forceinline__ double box_coord(double x, const double *__restrict__ ctr, const double *__restrict__ rad, int i) {
    return (x - ctr[i]) / rad[i];
}
__device__ __forceinline__ float box_coord(float x, const double *, const float *__restrict__ rad, int i) {
    return x * (1.f / rad[i]);
}

// The whole upward pass in one launch.  A CTA makes one leaf's multipole; the CTA that completes the last
// non-empty child of a node goes on with that node, so nothing waits and no level is a launch of its own.
// count[node] holds the children done and is zero again when the node has been taken.
// P2M: a thread sums one line of p coefficients (component, y, z) over the points, P2M's points shared by G groups
// where the lines are few.  M2M: the eight children are folded along z, y, x (8 -> 4 -> 2 -> 1 arrays: 14 line
// products where child by child takes 24).
// FP32, 2,000 atoms (419,000 points, 15,417 nodes, six levels): 0.39 -> 0.12 ms a product; FP64: 1.82 -> 1.01.
template <class T, int P, int NC>
__global__ void __launch_bounds__(Shape<T, P, NC>::UP_T)
    k_up(const ChebTables *__restrict__ tab, const int *__restrict__ leaves, const int *__restrict__ sb,
         const int *__restrict__ se, const double *__restrict__ ctr, const T *__restrict__ rad, const T *__restrict__ x,
         const T *__restrict__ y, const T *__restrict__ z, const T *__restrict__ dens, long ns, const int *__restrict__ nup,
         const int *__restrict__ parent, const int *__restrict__ child_first, const int *__restrict__ empty, int *count,
         T *mult) {
    using SH = Shape<T, P, NC>;
    constexpr int NL = SH::NL, N = SH::N, R = SH::R, PX = SH::PX, NT = SH::UP_T, G = SH::G;
    using RowT = Row<T, P, PX>;
    extern __shared__ __align__(16) unsigned char smem_up[];
    __shared__ RowT S[2][P];
    __shared__ Interp<T, P> I;
    __shared__ int last_s;
    const int tid = threadIdx.x;
    load_transfer<T, P, PX, false>(S, tab);
    I.load(tab);
    int node = leaves[blockIdx.x];
    {
        RowT *Sx = reinterpret_cast<RowT *>(smem_up);
        T(*Sy)[P] = reinterpret_cast<T(*)[P]>(Sx + 32);
        T(*Sz)[P] = Sy + 32;
        T(*D)[NC] = reinterpret_cast<T(*)[NC]>(Sz + 32);
        const int b = sb[node], e = se[node];
        const int g = tid / NL, r = tid % NL, d = r / (P * P), l = r / P % P, j = r % P;
        T acc[P] = {};
        __syncthreads();
        for (int base = b; base < e; base += 32) {
            const int cnt = min(32, e - base);
            if (tid < 96) {
                const int pt = tid & 31, ax = tid >> 5;
                if (pt < cnt) {
                    const T *X = ax == 0 ? x : (ax == 1 ? y : z);
                    I.at(box_coord(X[base + pt], ctr, rad, 3 * node + ax), [&](int m, T v) {
                        if (ax == 0) Sx[pt].v[m] = v;
                        else (ax == 1 ? Sy : Sz)[pt][m] = v;
                    });
                }
            } else if (tid < 128) {
                const int pt = tid - 96;
                if (pt < cnt)
                    for (int c = 0; c < NC; ++c) D[pt][c] = dens[c * ns + base + pt];
            }
            __syncthreads();
            if (g < G)
                for (int pt = g; pt < cnt; pt += G) {
                    const T w = Sy[pt][j] * Sz[pt][l] * D[pt][d];
                    const RowT s = Sx[pt];
#pragma unroll
                    for (int i = 0; i < P; ++i) acc[i] = fma(w, s.v[i], acc[i]);
                }
            __syncthreads();
        }
        T *red = reinterpret_cast<T *>(smem_up);  // [G][N]
        if (g < G)
#pragma unroll
            for (int i = 0; i < P; ++i) red[g * N + r * P + i] = acc[i];
        __syncthreads();
        for (int o = tid; o < N; o += NT) {
            T v = red[o];
#pragma unroll
            for (int q = 1; q < G; ++q) v += red[q * N + o];
            mult[(long)node * N + o] = v;
        }
    }
    T *A = reinterpret_cast<T *>(smem_up), *B = A + 4 * N;  // [4][N], [2][N]
    for (;;) {
        const int need = nup[node];  // the parent's children with sources; 0: nobody reads the parent
        if (need == 0) return;
        const int par = parent[node];
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            last_s = atomicAdd(count + par, 1) == need - 1;
            if (last_s) count[par] = 0;
            __threadfence();
        }
        __syncthreads();
        if (!last_s) return;
        const int c0 = child_first[par];
        // the children were written by other SMs during this launch: read through L2
        for (int q = tid; q < 4 * NL; q += NT) {
            const int c4 = q / NL, r = q % NL, off = r / (P * P) * R + r % (P * P);
            T out[P] = {};
#pragma unroll
            for (int zb = 0; zb < 2; ++zb) {
                const int ch = c0 + c4 + 4 * zb;
                if (empty[ch]) continue;
                T in[P];
#pragma unroll
                for (int k = 0; k < P; ++k) in[k] = __ldcg(mult + (long)ch * N + off + k * P * P);
                line<T, P, PX>(in, S[zb], out);
            }
#pragma unroll
            for (int k = 0; k < P; ++k) A[c4 * N + off + k * P * P] = out[k];
        }
        __syncthreads();
        for (int q = tid; q < 2 * NL; q += NT) {
            const int xb = q / NL, r = q % NL, off = r / P * (P * P) + r % P;
            T out[P] = {};
#pragma unroll
            for (int yb = 0; yb < 2; ++yb) {
                T in[P];
#pragma unroll
                for (int k = 0; k < P; ++k) in[k] = A[(xb + 2 * yb) * N + off + k * P];
                line<T, P, PX>(in, S[yb], out);
            }
#pragma unroll
            for (int k = 0; k < P; ++k) B[xb * N + off + k * P] = out[k];
        }
        __syncthreads();
        for (int q = tid; q < NL; q += NT) {
            T out[P] = {};
#pragma unroll
            for (int xb = 0; xb < 2; ++xb) {
                T in[P];
#pragma unroll
                for (int k = 0; k < P; ++k) in[k] = B[xb * N + q * P + k];
                line<T, P, PX>(in, S[xb], out);
            }
#pragma unroll
            for (int k = 0; k < P; ++k) mult[(long)par * N + q * P + k] = out[k];
        }
        node = par;
    }
}

// L2L, one parent a CTA: its local unfolded along x, y, z (1 -> 2 -> 4 -> 8 arrays) onto the children with
// targets (14 line products a parent where child by child takes 24).  FP32, 2,000 atoms: 0.12 -> 0.05 ms for the three
// levels; FP64, beside the near field: 1.66 -> 1.27.
constexpr int DOWN_T = 256;
template <class T, int P, int NC>
__global__ void __launch_bounds__(DOWN_T) k_down(const ChebTables *__restrict__ tab, const int *__restrict__ parents,
                                                 const int *__restrict__ child_first, const int *__restrict__ tb,
                                                 const int *__restrict__ te, T *local) {
    using SH = Shape<T, P, NC>;
    constexpr int NL = SH::NL, N = SH::N, R = SH::R, PX = SH::PX;
    extern __shared__ __align__(16) unsigned char smem_down[];
    __shared__ Row<T, P, PX> S[2][P];
    load_transfer<T, P, PX, true>(S, tab);
    const int par = parents[blockIdx.x], c0 = child_first[par], tid = threadIdx.x;
    T *A = reinterpret_cast<T *>(smem_down), *B = A + 4 * N;
    __syncthreads();
    for (int q = tid; q < NL; q += DOWN_T) {
        T in[P];
#pragma unroll
        for (int k = 0; k < P; ++k) in[k] = local[(long)par * N + q * P + k];
#pragma unroll
        for (int xb = 0; xb < 2; ++xb) {
            T out[P] = {};
            line<T, P, PX>(in, S[xb], out);
#pragma unroll
            for (int k = 0; k < P; ++k) B[xb * N + q * P + k] = out[k];
        }
    }
    __syncthreads();
    for (int q = tid; q < 2 * NL; q += DOWN_T) {
        const int xb = q / NL, r = q % NL, off = r / P * (P * P) + r % P;
        T in[P];
#pragma unroll
        for (int k = 0; k < P; ++k) in[k] = B[xb * N + off + k * P];
#pragma unroll
        for (int yb = 0; yb < 2; ++yb) {
            T out[P] = {};
            line<T, P, PX>(in, S[yb], out);
#pragma unroll
            for (int k = 0; k < P; ++k) A[(xb + 2 * yb) * N + off + k * P] = out[k];
        }
    }
    __syncthreads();
    for (int q = tid; q < 8 * NL; q += DOWN_T) {
        const int c8 = q / NL, r = q % NL, off = r / (P * P) * R + r % (P * P), ch = c0 + c8;
        if (tb[ch] >= te[ch]) continue;
        T in[P], out[P];
        T *dst = local + (long)ch * N + off;
#pragma unroll
        for (int k = 0; k < P; ++k) out[k] = dst[k * P * P];
#pragma unroll
        for (int k = 0; k < P; ++k) in[k] = A[(c8 & 3) * N + off + k * P * P];
        line<T, P, PX>(in, S[c8 >> 2], out);
#pragma unroll
        for (int k = 0; k < P; ++k) dst[k * P * P] = out[k];
    }
}

// L2P, one target leaf (of gridDim.y warps) a warp, a target a lane: summed line by line along x (one multiply-add a coefficient and
// component), added to the near field's sums already in out.  Leaves hold some 30 points: with a CTA of 128
// threads each, three of its four warps had none.
// FP32, 2,000 atoms: 0.108 -> 0.066 ms; FP64: 1.06 -> 0.89.
template <class T, int P, int NC>
__global__ void __launch_bounds__(32 * Shape<T, P, NC>::L2P_W)
    k_l2p(const ChebTables *__restrict__ tab, int nleaf, const int *__restrict__ tleaf, const int *__restrict__ tb_,
          const int *__restrict__ te_, const double *__restrict__ ctr, const T *__restrict__ rad, const T *__restrict__ tx,
          const T *__restrict__ ty, const T *__restrict__ tz, long nt, const T *__restrict__ local, double *out) {
    using SH = Shape<T, P, NC>;
    struct alignas(sizeof(T) * NC >= 16 ? 16 : sizeof(T) * NC) Vec {
        T v[NC];
    };
    extern __shared__ __align__(16) unsigned char smem_l2p[];
    __shared__ Interp<T, P> I;
    I.load(tab);
    const int k = blockIdx.x * SH::L2P_W + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int leaf = k < nleaf ? tleaf[k] : 0;
    const int tb = tb_[leaf] + 32 * blockIdx.y, te = k < nleaf ? te_[leaf] : 0;
    Vec *L = reinterpret_cast<Vec *>(smem_l2p) + (threadIdx.x >> 5) * SH::R;
    if (tb < te)
        for (int i = lane; i < SH::N; i += 32) L[i % SH::R].v[i / SH::R] = local[(long)leaf * SH::N + i];
    __syncthreads();
    for (int t = tb + lane; t < te; t += 32 * gridDim.y) {
        asm volatile("" ::: "memory");
        T w[3][P];
        I.at(box_coord(tx[t], ctr, rad, 3 * leaf), [&](int m, T v) { w[0][m] = v; });
        I.at(box_coord(ty[t], ctr, rad, 3 * leaf + 1), [&](int m, T v) { w[1][m] = v; });
        I.at(box_coord(tz[t], ctr, rad, 3 * leaf + 2), [&](int m, T v) { w[2][m] = v; });
        T acc[NC] = {};
#pragma unroll
        for (int c2 = 0; c2 < P; ++c2) {
            asm volatile("" ::: "memory");  // the coefficients stay in shared memory, not in (too many) registers
#pragma unroll
            for (int c1 = 0; c1 < P; ++c1) {
                T s[NC] = {};
#pragma unroll
                for (int c0 = 0; c0 < P; ++c0) {
                    const Vec c = L[(c2 * P + c1) * P + c0];
#pragma unroll
                    for (int o = 0; o < NC; ++o) s[o] = fma(w[0][c0], c.v[o], s[o]);
                }
                const T w12 = w[1][c1] * w[2][c2];
#pragma unroll
                for (int o = 0; o < NC; ++o) acc[o] = fma(w12, s[o], acc[o]);
            }
        }
#pragma unroll
        for (int o = 0; o < NC; ++o) out[o * nt + t] += (double)acc[o];
    }
}

// f(order) with the order as a compile-time constant
template <class F> void with_order(int p, F f) {
    switch (p) {
        case 2: f(std::integral_constant<int, 2>()); break;
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 5: f(std::integral_constant<int, 5>()); break;
        case 6: f(std::integral_constant<int, 6>()); break;
        case 7: f(std::integral_constant<int, 7>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        default: throw Error(IBIM_ERR_INVALID_ARGUMENT, "Chebyshev order out of range");
    }
}

template <class T, int P, int NC> void prepare() {
    using SH = Shape<T, P, NC>;
    static std::atomic<uint64_t> split, big;
    side_by_side(split, {(const void *)k_up<T, P, NC>, (const void *)k_down<T, P, NC>, (const void *)k_l2p<T, P, NC>});
    int dev = 0;
    IBIM_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (big.load() & bit) return;
    // above the 48 KB default, which the static tables count towards
    IBIM_CUDA(cudaFuncSetAttribute(k_up<T, P, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::SMEM));
    IBIM_CUDA(cudaFuncSetAttribute(k_down<T, P, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::UP_SMEM));
    IBIM_CUDA(cudaFuncSetAttribute(k_l2p<T, P, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   SH::L2P_W * SH::N * (int)sizeof(T)));
    big.fetch_or(bit);
}

template <class T, int NC>
void up(Plan &P, const T *rad, const T *x, const T *y, const T *z, const T *dens, T *mult) {
    if (P.np2m == 0) return;
    with_order(P.p, [&](auto order) {
        constexpr int O = decltype(order)::value;
        using SH = Shape<T, O, NC>;
        prepare<T, O, NC>();
        (count_launch(), k_up<T, O, NC><<<P.np2m, SH::UP_T, SH::SMEM, P.ctx->stream>>>(
            P.tables.ptr, P.p2m_nodes.ptr, P.nsrc_begin.ptr, P.nsrc_end.ptr, P.ncenter.ptr, rad, x, y, z, dens, P.ns,
            P.up_need.ptr, P.nparent.ptr, P.nchild_first.ptr, P.nempty.ptr, P.up_count.ptr, mult));
    });
    IBIM_CHECK_LAUNCH();
}

template <class T, int NC> void down(Plan &P, const TargetSet &S, T *local) {
    with_order(P.p, [&](auto order) {
        constexpr int O = decltype(order)::value;
        prepare<T, O, NC>();
        for (int l = 3; l < P.tree.nlevels; ++l) {
            const int b = S.l2l_level_begin[l], e = S.l2l_level_begin[l + 1];
            if (e > b)
                (count_launch(), k_down<T, O, NC><<<e - b, DOWN_T, Shape<T, O, NC>::UP_SMEM, P.ctx->stream>>>(
                    P.tables.ptr, S.l2l_parents.ptr + b, P.nchild_first.ptr, S.tbeg.ptr, S.tend.ptr, local));
        }
    });
    IBIM_CHECK_LAUNCH();
}

template <class T, int NC>
void l2p(Plan &P, const TargetSet &S, const T *rad, const T *tx, const T *ty, const T *tz, const T *local, double *out) {
    if (S.ntleaves == 0) return;
    with_order(P.p, [&](auto order) {
        constexpr int O = decltype(order)::value;
        using SH = Shape<T, O, NC>;
        prepare<T, O, NC>();
        // warps a leaf: as the average leaf fills; while they do not fill the device, as the largest leaf has
        // targets for (60 atoms, leaves of up to 128: 26 us with one warp, 16 with four; 2,000 atoms with leaves
        // of 36 on average: 0.061 ms with one, 0.079 with two)
        const int avg = std::max(1L, S.nt / S.ntleaves / 32), most = div_up(std::min(P.maxpoint, 256), 32);
        const int per = std::min(8, S.ntleaves <= 4 * P.ctx->num_sms ? std::max(avg, most) : avg);
        (count_launch(), k_l2p<T, O, NC><<<dim3(div_up(S.ntleaves, SH::L2P_W), per), 32 * SH::L2P_W,
                                           SH::L2P_W * SH::N * sizeof(T), P.ctx->stream>>>(P.tables.ptr, S.ntleaves, S.tleaf.ptr, S.tbeg.ptr, S.tend.ptr,
                                                            P.ncenter.ptr, rad, tx, ty, tz, S.nt, local, out));
    });
    IBIM_CHECK_LAUNCH();
}

}  // namespace

void translate_up(Plan &P, int nc, const double *dens, double *mult) {
    ProfScope ps_(PROF_P2M, 2.0 * nc * P.R * P.ns, 8.0 * (3 + nc) * P.ns);
    if (nc == 4) up<double, 4>(P, P.nradius.ptr, P.sx.ptr, P.sy.ptr, P.sz.ptr, dens, mult);
    else up<double, 1>(P, P.nradius.ptr, P.sx.ptr, P.sy.ptr, P.sz.ptr, dens, mult);
}
void translate_up(Plan &P, const float *dens, float *mult) {
    ProfScope ps_(PROF_P2M, 8.0 * P.R * P.ns, 28.0 * P.ns);
    up<float, 4>(P, P.nrad32.ptr, P.sxf.ptr, P.syf.ptr, P.szf.ptr, dens, mult);
}
void translate_down(Plan &P, const TargetSet &S, int nc, double *local) {
    ProfScope ps_(PROF_L2L);
    if (nc == 4) down<double, 4>(P, S, local);
    else down<double, 1>(P, S, local);
}
void translate_down(Plan &P, const TargetSet &S, float *local) {
    ProfScope ps_(PROF_L2L);
    down<float, 4>(P, S, local);
}
void translate_l2p(Plan &P, const TargetSet &S, int nc, const double *tx, const double *ty, const double *tz,
                   const double *local, double *out) {
    ProfScope ps_(PROF_L2P64, 2.0 * nc * P.R * S.nt, 8.0 * nc * P.R * S.ntleaves + (24.0 + 16.0 * nc) * S.nt);
    if (nc == 4) l2p<double, 4>(P, S, P.nradius.ptr, tx, ty, tz, local, out);
    else l2p<double, 1>(P, S, P.nradius.ptr, tx, ty, tz, local, out);
}
void translate_l2p(Plan &P, const TargetSet &S, const float *tx, const float *ty, const float *tz, const float *local,
                   double *out) {
    ProfScope ps_(PROF_L2P, 8.0 * P.R * S.nt, 16.0 * P.R * S.ntleaves + 76.0 * S.nt);
    l2p<float, 4>(P, S, P.nrad32.ptr, tx, ty, tz, local, out);
}

}  // namespace ibim
