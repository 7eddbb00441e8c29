// mw_kernels.cu -- sm_100a kernels of the MW apply: projection and two-scale transforms, norms, tree
// bookkeeping (Morton keys, hash index, splits), candidate screening, generated input nodes and the
// FP64 non-standard-form contraction.
//
// Node blocks are (2k)^3 FP64 tensors, x fastest; a node's transforms run on the FP64 matrix instruction, in place in
// shared memory (mw_block.cuh).
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdio>

#include "mw_block.cuh"
#include "mw_device.cuh"
#include "mw_kernels.cuh"

namespace mwb {

__global__ void k_hash_reset(uint64_t* hk, int* hv, uint32_t cap) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
        hk[i] = kEmptyKey;
        hv[i] = -1;
    }
}
// node i with key `key` into the open-addressing index (linear probing, at most cap probes)
__device__ __forceinline__ void hash_insert_one(uint64_t* hk, int* hv, uint32_t cap, uint64_t key, int i) {
    const uint32_t mask = cap - 1;
    uint32_t h = hslot(key, mask);
    for (uint32_t p = 0; p < cap; ++p) {
        unsigned long long old = atomicCAS((unsigned long long*)&hk[h], (unsigned long long)kEmptyKey,
                                           (unsigned long long)key);
        if (old == kEmptyKey || old == key) {
            hv[h] = i;
            return;
        }
        h = (h + 1) & mask;
    }
}
__global__ void k_hash_insert(uint64_t* hk, int* hv, uint32_t cap, const uint64_t* keys, int begin, int end) {
    const int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    hash_insert_one(hk, hv, cap, keys[i], i);
}

// ---------------------------------------------------------------------------------------------
// analytic functions (projection input)
// ---------------------------------------------------------------------------------------------

// hydrogen-like orbital (restated from reference src/analyticfunctions/HydrogenFunction.cpp:28-160)
__device__ inline double hydrogen(int n, int l, int m, double Z, double x, double y, double z) {
    double c = 0.0;
    if (n == 1 && l == 0) c = 2.0;
    else if (n == 2 && l == 0) c = 1.0 / (2.0 * sqrt(2.0));
    else if (n == 3 && l == 0) c = 1.0 / (9.0 * sqrt(3.0));
    else if (n == 2 && l == 1) c = 1.0 / (2.0 * sqrt(6.0));
    else if (n == 3 && l == 1) c = 1.0 / (9.0 * sqrt(6.0));
    else if (n == 3 && l == 2) c = 1.0 / (9.0 * sqrt(30.0));
    const double c0 = c * pow(Z, 1.5), c1 = 2.0 * Z / n;
    double a = 0.0;
    if (l == 0) a = 1.0;
    else if (l == 1) a = sqrt(3.0);
    else if (l == 2) a = (m <= 2) ? sqrt(15.0) : (m == 3 ? sqrt(15.0 / 4.0) : sqrt(5.0 / 4.0));
    const double ca = a / (2.0 * sqrt(3.14159265358979323846));
    const double rr = sqrt(x * x + y * y + z * z);
    const double rho = c1 * rr;
    double poly = 0.0;
    if (n == 1 && l == 0) poly = 1.0;
    else if (n == 2 && l == 0) poly = 2.0 - rho;
    else if (n == 3 && l == 0) poly = 6.0 - 6.0 * rho + rho * rho;
    else if (n == 2 && l == 1) poly = rho;
    else if (n == 3 && l == 1) poly = rho * (4.0 - rho);
    else if (n == 3 && l == 2) poly = rho * rho;
    const double radial = c0 * poly * exp(-0.5 * rho);
    double ang = 1.0;
    if (l == 1) {
        if (rr == 0.0) return 0.0;
        ang = (m == 0 ? x : (m == 1 ? y : z)) / rr;
    } else if (l == 2) {
        if (rr == 0.0) return 0.0;
        const double r2 = rr * rr;
        if (m == 0) ang = x * y / r2;
        else if (m == 1) ang = x * z / r2;
        else if (m == 2) ang = y * z / r2;
        else if (m == 3) ang = (x * x - y * y) / r2;
        else ang = (2.0 * z * z - x * x - y * y) / r2;
    }
    return radial * ca * ang;
}

// products of hydrogen orbitals (Gaussian sums are evaluated by their factors, transform_node)
__device__ inline double eval_func(const FuncDesc& f, double x, double y, double z) {
    double v = 0.0;
    if (f.type == 2) {
        for (int t = 0; t < f.nterm; ++t) {
            const double* q = f.p + 1 + 11 * t;
            const double X = x - q[8], Y = y - q[9], Zc = z - q[10];
            double a = hydrogen((int)q[1], (int)q[2], (int)q[3], q[7], X, Y, Zc);
            double b = ((int)q[4] > 0) ? hydrogen((int)q[4], (int)q[5], (int)q[6], q[7], X, Y, Zc) : 1.0;
            v += q[0] * a * b;
        }
    }
    return v;
}

// ---------------------------------------------------------------------------------------------
// projection / compression / sum-up of node blocks
// ---------------------------------------------------------------------------------------------

struct TView {
    uint64_t* key;
    int* parent;
    int* child0;
    double* coef;
    double* norm2;
    double* wnorm2;
};
inline TView view(Tree& t) { return TView{t.key, t.parent, t.child0, t.coef, t.norm2, t.wnorm2}; }

struct WorldGeo {
    int n0;
    double lo[3];  // world corner (physical)
    double qx[16]; // quadrature nodes on [0,1]
};

constexpr int kGaussBatch = 8;

template <int K>
struct TrCfg {
    using B = BX<K, 2 * K>;
    static constexpr size_t SMEM = sizeof(double) * (B::VOL + 2 * B::FRAG);
    static constexpr int MINB = K <= 6 ? 4 : K <= 10 ? 2 : 1;  // blocks per SM (registers and shared memory)
};

// One node of a transform (the whole block); leaves must have been filtered out by the caller in the compress /
// sum-up modes.  fr: the operator's fragments.  HBM- and FP64-bound in like parts (k = 10: 128 KB of traffic and 18,000 cycles
// of products per node and SM); with a thread per pencil the level of 16 trees took twice as long.
template <int K>
__device__ __forceinline__ void transform_node(int mode, int node, const TView& t, const double* __restrict__ fr,
                                               const FuncDesc& f, const WorldGeo& wg) {
    using B = BX<K, 2 * K>;
    constexpr int K2 = 2 * K, BS = Geo<K>::BS;
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[64];
    __shared__ double gf[kGaussBatch][3][K2];
    double* X = sm;
    double* fo = X + B::VOL;
    bx_operator(fo, fr, 2 * B::FRAG, B::NTHR);
    auto at = [](int a, int b, int c) { return a + B::LDA * b + B::LDP * c; };
    double fac = 1.0;
    if (mode == TM_PROJECT) {
        long long tr[3];
        const uint64_t key = t.key[node];
        key_trans(key, tr);
        const int n1 = wg.n0 + key_depth(key) + 1;
        const double h = ldexp(1.0, -n1);
        fac = pow(2.0, -1.5 * n1);
        auto coord = [&](int d, int i) { return wg.lo[d] + (2 * tr[d] + i / K + wg.qx[i % K]) * h; };
        if (f.type == 1) {
            // sums of Gaussians: the factors along each direction once per node (3 x 2k exponentials per Gaussian instead
            // of (2k)^3; they were most of a projection), eight Gaussians at a time
            for (int g0 = 0; g0 < f.nterm; g0 += kGaussBatch) {
                const int ng = min(kGaussBatch, f.nterm - g0);
                if (g0 > 0) __syncthreads();  // the previous factors are read
                for (int e = threadIdx.x; e < ng * 3 * K2; e += B::NTHR) {
                    const int g = e / (3 * K2), d = (e / K2) % 3, i = e % K2;
                    const double* q = f.p + 1 + 8 * (g0 + g);
                    const double u = coord(d, i) - q[2 + d];
                    double v = d == 0 ? q[0] : 1.0;
                    for (int j = 0; j < (int)q[5 + d]; ++j) v *= u;
                    gf[g][d][i] = v * exp(-q[1] * u * u);
                }
                __syncthreads();
                for (int e = threadIdx.x; e < BS; e += B::NTHR) {
                    const int a = e % K2, b = (e / K2) % K2, c = e / (K2 * K2);
                    double v = g0 > 0 ? X[at(a, b, c)] : 0.0;
                    for (int g = 0; g < ng; ++g) v = fma(gf[g][0][a] * gf[g][1][b], gf[g][2][c], v);
                    X[at(a, b, c)] = v;
                }
            }
            if (f.nterm <= 0)
                for (int e = threadIdx.x; e < B::VOL; e += B::NTHR) X[e] = 0.0;
        } else {
            for (int e = threadIdx.x; e < BS; e += B::NTHR) {
                const int a = e % K2, b = (e / K2) % K2, c = e / (K2 * K2);
                X[at(a, b, c)] = eval_func(f, coord(0, a), coord(1, b), coord(2, c));
            }
        }
    } else if (mode == TM_COMPRESS) {
        const int c0 = t.child0[node];
        // the children's scaling rows; element pairs by asynchronous copies where a pair never straddles children
        constexpr int W = K % 2 == 0 ? 2 : 1;
        for (int e = threadIdx.x; e < BS / W; e += B::NTHR) {
            const int a = W * (e % (K2 / W)), b = (e / (K2 / W)) % K2, c = e / (K2 / W * K2);
            const int ch = (a / K) + 2 * (b / K) + 4 * (c / K);
            const double* src = t.coef + (size_t)(c0 + ch) * BS + (a % K) + K2 * ((b % K) + K2 * (c % K));
            if constexpr (W == 2) cp_async16(X + at(a, b, c), src);
            else X[at(a, b, c)] = *src;
        }
    } else {
        bx_load<K, B::NWARP>(X, t.coef + (size_t)node * BS);
    }
    cp_async_wait_all();
    __syncthreads();
    bx_slices<K, 2 * K>(X, fo, fo + B::FRAG);
    __syncthreads();
    double n2 = 0.0, w2 = 0.0;
    const int c0 = (mode == TM_SUMUP) ? t.child0[node] : 0;
    bx_columns<K, 2 * K>(X, fo, [&](int c, int n, double v0, double v1) {
        const int a = n % K2, b = n / K2;
        if (mode == TM_SUMUP) {
            const int ch = 2 * (b / K) + 4 * (c / K), in = K2 * ((b % K) + K2 * (c % K));
            if constexpr (K % 2 == 0) {
                double2* p = reinterpret_cast<double2*>(t.coef + (size_t)(c0 + ch + a / K) * BS + a % K + in);
                const double2 o = *p;
                *p = make_double2(o.x + v0, o.y + v1);
            } else {
                t.coef[(size_t)(c0 + ch + a / K) * BS + a % K + in] += v0;
                t.coef[(size_t)(c0 + ch + (a + 1) / K) * BS + (a + 1) % K + in] += v1;
            }
        } else {
            v0 *= fac;
            v1 *= fac;
            *reinterpret_cast<double2*>(t.coef + (size_t)node * BS + n + K2 * K2 * c) = make_double2(v0, v1);
            n2 += v0 * v0 + v1 * v1;
            const bool sc = b < K && c < K;
            if (!(sc && a < K)) w2 += v0 * v0;
            if (!(sc && a + 1 < K)) w2 += v1 * v1;
        }
    });
    if (mode != TM_SUMUP) {
        block_sum2(n2, w2, red);
        if (threadIdx.x == 0) {
            t.norm2[node] = n2;
            t.wnorm2[node] = w2;
        }
    }
}

template <int K>
__global__ void __launch_bounds__(BX<K, 2 * K>::NTHR, TrCfg<K>::MINB)
    k_transform(int mode, const int* __restrict__ nodes, int begin, TView t, const double* __restrict__ fr, FuncDesc f, WorldGeo wg) {
    // node list, or (nodes == nullptr) the range begin + blockIdx.x, where leaves have nothing to do
    // for the compress / sum-up modes (the whole block leaves together, before any barrier)
    const int node = nodes ? nodes[blockIdx.x] : begin + blockIdx.x;
    if (!nodes && mode != TM_PROJECT && t.child0[node] < 0) return;
    transform_node<K>(mode, node, t, fr, f, wg);
}

// compress / sum-up of the internal nodes of one level of several trees: items (tree, node)
template <int K>
__global__ void __launch_bounds__(BX<K, 2 * K>::NTHR, TrCfg<K>::MINB)
    k_transform_multi(int mode, const int2* __restrict__ items, const TView* __restrict__ views, const double* __restrict__ fr, WorldGeo wg) {
    const int2 it = items[blockIdx.x];
    const TView t = views[it.x];
    if (t.child0[it.y] < 0) return;
    transform_node<K>(mode, it.y, t, fr, FuncDesc{0, 0, nullptr}, wg);
}

// one warp per (tree, node) item: squared norm of the block and of its wavelet part
template <int K>
__global__ void k_node_norms_multi(const int2* __restrict__ items, int nitems, const TView* __restrict__ views) {
    using G = Geo<K>;
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (q >= nitems) return;
    const int2 it = items[q];
    const TView t = views[it.x];
    const double* c = t.coef + (size_t)it.y * G::BS;
    double n2 = 0.0, w2 = 0.0;
    for (int e = lane; e < G::BS; e += 32) {
        const double v = c[e];
        const int a = e % G::K2, b = (e / G::K2) % G::K2, cc = e / (G::K2 * G::K2);
        n2 += v * v;
        if (!(a < K && b < K && cc < K)) w2 += v * v;
    }
    for (int o = 16; o; o >>= 1) {
        n2 += __shfl_down_sync(0xffffffffu, n2, o);
        w2 += __shfl_down_sync(0xffffffffu, w2, o);
    }
    if (lane == 0) {
        t.norm2[it.y] = n2;
        t.wnorm2[it.y] = w2;
    }
}

// one warp per node: squared norm of the block and of its wavelet part
template <int K>
__global__ void k_node_norms(TView t, int begin, int end) {
    using G = Geo<K>;
    const int node = begin + (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (node >= end) return;
    const double* c = t.coef + (size_t)node * G::BS;
    double n2 = 0.0, w2 = 0.0;
    for (int e = lane; e < G::BS; e += 32) {
        const double v = c[e];
        const int a = e % G::K2, b = (e / G::K2) % G::K2, cc = e / (G::K2 * G::K2);
        n2 += v * v;
        if (!(a < K && b < K && cc < K)) w2 += v * v;
    }
    for (int o = 16; o; o >>= 1) {
        n2 += __shfl_down_sync(0xffffffffu, n2, o);
        w2 += __shfl_down_sync(0xffffffffu, w2, o);
    }
    if (lane == 0) {
        t.norm2[node] = n2;
        t.wnorm2[node] = w2;
    }
}

// children of the split nodes of several trees in one launch: entry q of the flat list belongs to tree
// tree_of[q]; its 8 children are appended after the tree's first nold nodes (in list order) and
// entered into the tree's hash index
struct ChildTree {
    TView t;
    uint64_t* hkey;
    int* hval;
    uint32_t hcap;
    int nold;   // nodes before the appended children
    int first;  // first list entry of this tree
};
__global__ void k_make_children_many(const ChildTree* __restrict__ ts, const int* __restrict__ tree_of,
                                     const int* __restrict__ list, int ntot) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ntot) return;
    const ChildTree& T = ts[tree_of[q]];
    const int p = list[q];
    const int c0 = T.nold + 8 * (q - T.first);
    T.t.child0[p] = c0;
    long long tr[3];
    const uint64_t key = T.t.key[p];
    key_trans(key, tr);
    const int d = key_depth(key) + 1;
    for (int c = 0; c < 8; ++c) {
        const int i = c0 + c;
        const uint64_t ck = make_key(d, 2 * tr[0] + (c & 1), 2 * tr[1] + ((c >> 1) & 1), 2 * tr[2] + ((c >> 2) & 1));
        T.t.key[i] = ck;
        T.t.parent[i] = p;
        T.t.child0[i] = -1;
        T.t.norm2[i] = 0.0;
        T.t.wnorm2[i] = 0.0;
        hash_insert_one(T.hkey, T.hval, T.hcap, ck, i);
    }
}

// deterministic single-block reductions (fixed summation order)
__device__ __forceinline__ double reduce_norm2_block(const double* __restrict__ norm2, const int* __restrict__ child0,
                                                     int begin, int end, int leaves_only, int want_max) {
    __shared__ double red[64];
    double s = 0.0, dummy = 0.0;
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
        if (leaves_only && child0[i] >= 0) continue;
        s = want_max ? fmax(s, norm2[i]) : s + norm2[i];
    }
    if (want_max) {
        for (int o = 16; o; o >>= 1) s = fmax(s, __shfl_down_sync(0xffffffffu, s, o));
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (l == 0) red[w] = s;
        __syncthreads();
        if (w == 0) {
            s = l < (int)(blockDim.x >> 5) ? red[l] : 0.0;
            for (int o = 16; o; o >>= 1) s = fmax(s, __shfl_down_sync(0xffffffffu, s, o));
        }
    } else {
        block_sum2(s, dummy, red);
    }
    return s;
}
__global__ void k_reduce_norm2(const double* __restrict__ norm2, const int* __restrict__ child0, int begin,
                               int end, int leaves_only, int want_max, double* out) {
    const double s = reduce_norm2_block(norm2, child0, begin, end, leaves_only, want_max);
    if (threadIdx.x == 0) *out = s;
}
// both reductions of several trees in one launch: block b reduces tree b % nt, the leaf sum when
// b < nt, else the largest node norm (the same blocks as k_reduce_norm2, so the same sums)
struct NormSrc {
    const double* norm2;
    const int* child0;
    int n;
};
__global__ void k_reduce_norm2_many(const NormSrc* __restrict__ src, int nt, double* out) {
    const int t = blockIdx.x % nt, mx = blockIdx.x / nt;
    const NormSrc ns = src[t];
    const double s = reduce_norm2_block(ns.norm2, ns.child0, 0, ns.n, !mx, mx);
    if (threadIdx.x == 0) out[mx * nt + t] = s;
}

// Split decisions of a tree's last level in one block: the threshold from the leaves' norm (the same sum as
// k_reduce_norm2), then the level's nodes above it, in order.  fac = 2^{-depth / 2}; out[0] = count, list follows
__global__ void __launch_bounds__(1024) k_level_split(const double* __restrict__ norm2, const double* __restrict__ wnorm2,
                                                      const int* __restrict__ child0, int begin, int end, double prec,
                                                      double fac, int may_split, int* out) {
    __shared__ double thr;
    __shared__ int wsum[32];
    const double s2 = reduce_norm2_block(norm2, child0, 0, end, 1, 0);
    if (threadIdx.x == 0) thr = prec * sqrt(s2) * fac;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int b = begin; b < end; b += 1024) {
        const int i = b + threadIdx.x;
        const bool f = i < end && may_split && sqrt(wnorm2[i]) > thr;
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (f) out[1 + base + before + __popc(m & ((1u << lane) - 1u))] = i;
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = base;
}
// children of the listed nodes, appended after the first nold nodes and entered into the hash index
__global__ void k_make_children(TView t, uint64_t* hkey, int* hval, uint32_t hcap, const int* __restrict__ list, int nsplit, int nold) {
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) / 8, c = threadIdx.x & 7;
    if (q >= nsplit) return;
    const int p = list[q], i = nold + 8 * q + c;
    if (c == 0) t.child0[p] = nold + 8 * q;
    long long tr[3];
    const uint64_t key = t.key[p];
    key_trans(key, tr);
    const uint64_t ck = make_key(key_depth(key) + 1, 2 * tr[0] + (c & 1), 2 * tr[1] + ((c >> 1) & 1), 2 * tr[2] + ((c >> 2) & 1));
    t.key[i] = ck;
    t.parent[i] = p;
    t.child0[i] = -1;
    t.norm2[i] = 0.0;
    t.wnorm2[i] = 0.0;
    hash_insert_one(hkey, hval, hcap, ck, i);
}

__global__ void k_rescale(double* coef, size_t n, double c) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        coef[i] *= c;
}

// <a|b>: groups of four warps (so that a small block's loads are all in flight at once) take nodes of a in turn, the product
// over the wavelet part (all components at depth 0), then the last block to finish adds the groups' parts in a fixed order
// and writes the sum where the host reads it (mapped memory).  A second launch for the sum, a copy and two scalar loads per
// element took twice as long.  A part for every node made the last block's loop over them a large share of the call on trees
// of many small blocks, so below k = 8 the blocks are at most 8 per SM, whose groups take nodes in turn (64,000 nodes at
// k = 4 141 -> 66 us, 34,264 at k = 5 103 -> 63).  From k = 8 up a group takes one node: a node's loads keep the SM busy, and
// nodes in turn cost more than the loop saves (17,088 nodes at k = 10: 206 us, 258 in turn).
constexpr int kDotThreads = 256, kDotGroups = kDotThreads / 128;
constexpr bool dot_in_turn(int k) { return k < 8; }
template <int K>
__global__ void __launch_bounds__(kDotThreads) k_dot(TView a, int na, const double* __restrict__ bcoef, const uint64_t* hk,
                                                     const int* hv, uint32_t hcap, double* part, unsigned* ticket, double* out) {
    using G = Geo<K>;
    __shared__ double red[64];
    __shared__ unsigned done;
    __shared__ double ws[kDotThreads / 32];
    const int group = blockIdx.x * kDotGroups + threadIdx.x / 128, t = threadIdx.x & 127;
    const int nparts = dot_in_turn(K) ? min(na, (int)gridDim.x * kDotGroups) : na;
    double s = 0.0;
    for (int node = group; node < na; node += gridDim.x * kDotGroups) {
        const uint64_t key = a.key[node];
        const int j = hlookup(hk, hv, hcap, key);
        if (j >= 0) {
            const bool root = key_depth(key) == 0;
            const double2* x = reinterpret_cast<const double2*>(a.coef + (size_t)node * G::BS);
            const double2* y = reinterpret_cast<const double2*>(bcoef + (size_t)j * G::BS);
#pragma unroll 8
            for (int e = t; e < G::BS / 2; e += 128) {
                const double2 u = x[e], v = y[e];
                const int aa = 2 * (e % K), bb = (e / K) % G::K2, cc = e / (K * G::K2);
                const bool sc = !root && bb < K && cc < K;
                if (!(sc && aa < K)) s = fma(u.x, v.x, s);
                if (!(sc && aa + 1 < K)) s = fma(u.y, v.y, s);
            }
        }
        if constexpr (!dot_in_turn(K)) break;
    }
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (t == 0 && group < nparts) {
        const double* w = ws + (threadIdx.x >> 5);
        part[group] = (w[0] + w[1]) + (w[2] + w[3]);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) done = atomicAdd(ticket, 1u);
    __syncthreads();
    if (done != gridDim.x - 1) return;
    __threadfence();
    double d = 0.0;
    s = 0.0;
    for (int i = threadIdx.x; i < nparts; i += kDotThreads) s += __ldcg(part + i);
    block_sum2(s, d, red);
    if (threadIdx.x == 0) {
        *ticket = 0u;  // for the next call on this stream
        *out = s;
    }
}
// ||a - b||^2 contributions of a's nodes (one warp per node): root scaling parts and all wavelet
// parts of a - b, where b's node is missing its block counts as zero; with `only_missing` the
// nodes of a that b lacks alone (the second half of the sum, run with the roles swapped)
template <int K>
__global__ void k_diff_nodes(TView a, int na, const double* __restrict__ bcoef, const uint64_t* hk, const int* hv,
                             uint32_t hcap, int only_missing, double* part) {
    using G = Geo<K>;
    const int node = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (node >= na) return;
    const uint64_t key = a.key[node];
    const int j = hlookup(hk, hv, hcap, key);
    double s = 0.0;
    if (!(only_missing && j >= 0)) {
        const bool root = key_depth(key) == 0;
        const double* x = a.coef + (size_t)node * G::BS;
        const double* y = j >= 0 ? bcoef + (size_t)j * G::BS : nullptr;
        for (int e = lane; e < G::BS; e += 32) {
            const int aa = e % G::K2, bb = (e / G::K2) % G::K2, cc = e / (G::K2 * G::K2);
            if (!root && aa < K && bb < K && cc < K) continue;
            const double d = x[e] - (y ? y[e] : 0.0);
            s += d * d;
        }
    }
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) part[node] = s;
}
__global__ void k_sum_array(const double* __restrict__ v, int n, double* out) {
    __shared__ double red[64];
    double s = 0.0, d = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += v[i];
    block_sum2(s, d, red);
    if (threadIdx.x == 0) *out = s;
}

// ---------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------

static inline void count(Ctx* c, int n = 1) { c->launches += n; }

#define MWB_DISPATCH_K(k, F)                                    \
    switch (k) {                                                \
        case 4: F(4); break;                                    \
        case 5: F(5); break;                                    \
        case 6: F(6); break;                                    \
        case 7: F(7); break;                                    \
        case 8: F(8); break;                                    \
        case 9: F(9); break;                                    \
        case 10: F(10); break;                                  \
        case 11: F(11); break;                                  \
        case 12: F(12); break;                                  \
        default: throw Error(-1, "unsupported order (k must be 4..12)"); \
    }

static WorldGeo world_geo(const Mra& m) {
    WorldGeo g{};
    g.n0 = m.n0;
    for (int d = 0; d < 3; ++d) g.lo[d] = m.corner[d] * std::ldexp(1.0, -m.n0);
    for (int i = 0; i < m.k && i < 16; ++i) g.qx[i] = m.basis.qx[i];
    return g;
}

void world_fragments(Mra& m, const std::vector<double>& PF, const std::vector<double>& MV, const std::vector<double>& FT) {
    std::vector<double> f;
    const std::vector<double>* mats[4] = {&m.F, &FT, &PF, &MV};
#define L_FR(KK)                                                                            \
    {                                                                                       \
        constexpr int N = BX<KK, 2 * KK>::FRAG, W = 2 * KK;                                  \
        m.fr_n = N;                                                                          \
        f.resize(8 * N);                                                                     \
        for (int q = 0; q < 4; ++q) {                                                        \
            auto entry = [&](int o, int i) { return (*mats[q])[(size_t)o * W + i]; };        \
            for (int e = 0; e < N; ++e) {                                                    \
                f[2 * q * N + e] = bx_frag_a<KK, 2 * KK>(e, entry);                          \
                f[(2 * q + 1) * N + e] = bx_frag_b<KK, 2 * KK>(e, entry);                    \
            }                                                                                \
        }                                                                                    \
        constexpr int NH = BX<KK, KK>::FRAG;                                                 \
        f.resize(8 * N + 4 * NH);                                                            \
        for (int bit = 0; bit < 2; ++bit) {                                                  \
            auto entry = [&](int o, int i) { return FT[(size_t)(bit * KK + o) * W + i]; };   \
            for (int e = 0; e < NH; ++e) {                                                   \
                f[8 * N + 2 * bit * NH + e] = bx_frag_a<KK, KK>(e, entry);                   \
                f[8 * N + (2 * bit + 1) * NH + e] = bx_frag_b<KK, KK>(e, entry);             \
            }                                                                                \
        }                                                                                    \
    }
    MWB_DISPATCH_K(m.k, L_FR)
#undef L_FR
    m.d_frF = (double*)dalloc(m.ctx, sizeof(double) * f.size());  // one allocation for all
    m.d_frFT = m.d_frF + 2 * m.fr_n;
    m.d_frPF = m.d_frF + 4 * m.fr_n;
    m.d_frMV = m.d_frF + 6 * m.fr_n;
    m.d_frH = m.d_frF + 8 * m.fr_n;
    upload_bytes(m.ctx, m.d_frF, f.data(), sizeof(double) * f.size());
}

void launch_transform_nodes(Tree& t, int mode, const int* d_nodes, int nnodes, const FuncDesc* f, cudaStream_t s,
                            int begin) {
    if (nnodes <= 0) return;
    const Mra& m = *t.mra;
    const double* fr = (mode == TM_PROJECT) ? m.d_frPF : (mode == TM_COMPRESS ? m.d_frF : m.d_frFT);
    FuncDesc fd = f ? *f : FuncDesc{0, 0, nullptr};
    WorldGeo wg = world_geo(m);
    TView tv = view(t);
#define L_TR(KK)                                                                                              \
    {                                                                                                         \
        MWB_CUDA(cudaFuncSetAttribute(k_transform<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize,           \
                                      (int)TrCfg<KK>::SMEM));                                                 \
        k_transform<KK><<<nnodes, BX<KK, 2 * KK>::NTHR, TrCfg<KK>::SMEM, s>>>(mode, d_nodes, begin, tv, fr, fd, wg); \
    }
    MWB_DISPATCH_K(m.k, L_TR)
#undef L_TR
    MWB_CUDA(cudaGetLastError());
    count(m.ctx);
}

// Finishing transforms of a batch of trees on one world, one launch per level for all trees:
// sum-up top-down (sumup), then compress bottom-up, then the norms of every node (the sums an upload makes, so that a
// tree read back has them bit for bit).
void trees_finish(const std::vector<Tree*>& ts, bool sumup, cudaStream_t s) {
    if (ts.empty()) return;
    const Mra& m = *ts[0]->mra;
    Ctx* ctx = m.ctx;
    int maxl = 0;
    for (Tree* t : ts) maxl = std::max(maxl, t->levels());
    // items grouped by level: [lvl_off[d], lvl_off[d+1]) are the nodes of depth d of every tree
    std::vector<int2> items;
    std::vector<int> lvl_off(maxl + 1, 0);
    for (int d = 0; d < maxl; ++d) {
        lvl_off[d] = (int)items.size();
        for (size_t i = 0; i < ts.size(); ++i)
            if (d < ts[i]->levels())
                for (int q = ts[i]->level_begin[d]; q < ts[i]->level_begin[d + 1]; ++q) items.push_back(int2{(int)i, q});
    }
    lvl_off[maxl] = (int)items.size();
    if (items.empty()) return;
    std::vector<TView> views;
    for (Tree* t : ts) views.push_back(view(*t));
    UploadPack up(ctx);
    const size_t o_items = up.add(items), o_views = up.add(views);
    char* d_up = up.send();
    const int2* d_items = reinterpret_cast<const int2*>(d_up + o_items);
    const TView* d_views = reinterpret_cast<const TView*>(d_up + o_views);
    WorldGeo wg = world_geo(m);
    auto level = [&](int mode, int d) {
        const int n = lvl_off[d + 1] - lvl_off[d];
        if (n <= 0) return;
        const double* fr = mode == TM_COMPRESS ? m.d_frF : m.d_frFT;
#define L_TRM(KK)                                                                                          \
    {                                                                                                      \
        MWB_CUDA(cudaFuncSetAttribute(k_transform_multi<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                      (int)TrCfg<KK>::SMEM));                                              \
        k_transform_multi<KK><<<n, BX<KK, 2 * KK>::NTHR, TrCfg<KK>::SMEM, s>>>(mode, d_items + lvl_off[d], d_views, fr, wg); \
    }
        MWB_DISPATCH_K(m.k, L_TRM)
#undef L_TRM
        MWB_CUDA(cudaGetLastError());
        count(ctx);
    };
    if (sumup)
        for (int d = 0; d + 1 < maxl; ++d) level(TM_SUMUP, d);
    for (int d = maxl - 2; d >= 0; --d) level(TM_COMPRESS, d);
    {
        const int n = (int)items.size();
#define L_NNM(KK) k_node_norms_multi<KK><<<(n * 32 + 255) / 256, 256, 0, s>>>(d_items, n, d_views);
        MWB_DISPATCH_K(m.k, L_NNM)
#undef L_NNM
        MWB_CUDA(cudaGetLastError());
        count(ctx);
    }
    dfree(ctx, d_up);
}

void launch_node_norms(Tree& t, int begin, int end, cudaStream_t s) {
    if (end <= begin) return;
    const int n = end - begin;
    TView tv = view(t);
#define L_NN(KK) k_node_norms<KK><<<(n * 32 + 255) / 256, 256, 0, s>>>(tv, begin, end);
    MWB_DISPATCH_K(t.mra->k, L_NN)
#undef L_NN
    MWB_CUDA(cudaGetLastError());
    count(t.mra->ctx);
}

void launch_hash_reset(Tree& t, cudaStream_t s) {
    k_hash_reset<<<std::min<uint32_t>((t.hcap + 255) / 256, 4096), 256, 0, s>>>(t.hkey, t.hval, t.hcap);
    MWB_CUDA(cudaGetLastError());
    count(t.mra->ctx);
}
void launch_hash_insert(Tree& t, int begin, int end, cudaStream_t s) {
    if (end <= begin) return;
    k_hash_insert<<<(end - begin + 255) / 256, 256, 0, s>>>(t.hkey, t.hval, t.hcap, t.key, begin, end);
    MWB_CUDA(cudaGetLastError());
    count(t.mra->ctx);
}

// split the nodes of the tree's last level whose wavelet norm exceeds prec ||f|| 2^{-depth/2}; returns the number of
// new nodes (two launches and one read-back)
int tree_refine_last_level(Tree& t, double prec) {
    Ctx* ctx = t.mra->ctx;
    cudaStream_t s = ctx->stream;
    const int depth = t.levels() - 1, b = t.level_begin[depth], e = t.level_begin[depth + 1];
    int* d_out = (int*)dalloc(ctx, sizeof(int) * (e - b + 1));
    k_level_split<<<1, 1024, 0, s>>>(t.norm2, t.wnorm2, t.child0, b, e, prec, std::pow(2.0, -0.5 * depth),
                                     depth < t.mra->depth_limit, d_out);
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    int ns = 0;
    readback(ctx, {{&ns, d_out, sizeof(int)}});
    if (ns > 0) {
        tree_reserve(t, t.n + 8 * ns);
        k_make_children<<<(ns + 15) / 16, 128, 0, s>>>(view(t), t.hkey, t.hval, t.hcap, d_out + 1, ns, t.n);
        MWB_CUDA(cudaGetLastError());
        count(ctx);
        t.n += 8 * ns;
        t.level_begin.push_back(t.n);
    }
    dfree(ctx, d_out);
    return 8 * ns;
}

void trees_add_children(const std::vector<Tree*>& ts, const std::vector<std::vector<int>>& lists, cudaStream_t s) {
    size_t tot = 0;
    for (auto& l : lists) tot += l.size();
    if (tot == 0 || ts.empty()) return;
    Ctx* ctx = ts[0]->mra->ctx;
    std::vector<ChildTree> ct;
    std::vector<int> buf(2 * tot);  // list entries, then their tree (index into ct)
    size_t off = 0;
    for (size_t i = 0; i < ts.size(); ++i) {
        Tree& t = *ts[i];
        const int ns = (int)lists[i].size();
        if (ns == 0) continue;
        tree_reserve(t, t.n + 8 * ns);  // may move the arrays and grow the hash index
        ct.push_back(ChildTree{view(t), t.hkey, t.hval, t.hcap, t.n, (int)off});
        for (int q = 0; q < ns; ++q) {
            buf[off + q] = lists[i][q];
            buf[tot + off + q] = (int)ct.size() - 1;
        }
        off += ns;
    }
    UploadPack up(ctx);
    const size_t o_buf = up.add(buf), o_ct = up.add(ct);
    char* d_up = up.send();
    const int* d_buf = reinterpret_cast<const int*>(d_up + o_buf);
    const ChildTree* d_ct = reinterpret_cast<const ChildTree*>(d_up + o_ct);
    k_make_children_many<<<(int)((tot + 127) / 128), 128, 0, s>>>(d_ct, d_buf + tot, d_buf, (int)tot);
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    for (size_t i = 0; i < ts.size(); ++i) {
        Tree& t = *ts[i];
        const int ns = (int)lists[i].size();
        if (ns == 0) continue;
        t.n += 8 * ns;
        t.level_begin.push_back(t.n);
    }
    dfree(ctx, d_up);  // stream-ordered; the host vectors were staged
}

double reduce_leaf_norm2(Tree& t, cudaStream_t s) {
    if (t.n <= 0) return 0.0;
    Ctx* ctx = t.mra->ctx;
    double* d = (double*)dalloc(ctx, sizeof(double));
    k_reduce_norm2<<<1, 1024, 0, s>>>(t.norm2, t.child0, 0, t.n, 1, 0, d);
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    double h = 0.0;
    MWB_CUDA(cudaMemcpyAsync(&h, d, sizeof(double), cudaMemcpyDeviceToHost, s));
    MWB_CUDA(cudaStreamSynchronize(s));
    dfree(ctx, d);
    return h;
}

// squared norm (leaves) and largest node norm^2 of several trees with one synchronisation
void reduce_norms_many(const std::vector<Tree*>& ts, std::vector<double>& leaf2, std::vector<double>& max2,
                       cudaStream_t s) {
    const int n = (int)ts.size();
    leaf2.assign(n, 0.0);
    max2.assign(n, 0.0);
    if (n == 0) return;
    Ctx* ctx = ts[0]->mra->ctx;
    double* d = (double*)dalloc(ctx, sizeof(double) * 2 * n);
    std::vector<NormSrc> src(n);
    for (int i = 0; i < n; ++i) src[i] = NormSrc{ts[i]->norm2, ts[i]->child0, ts[i]->n};  // n = 0: zero sums
    NormSrc* d_src = (NormSrc*)dalloc(ctx, sizeof(NormSrc) * n);
    upload_bytes(ctx, d_src, src.data(), sizeof(NormSrc) * n);
    k_reduce_norm2_many<<<2 * n, 1024, 0, s>>>(d_src, n, d);
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    dfree(ctx, d_src);
    std::vector<double> h(2 * n);
    readback(ctx, {{h.data(), d, sizeof(double) * 2 * n}});  // on the context's stream (= s)
    dfree(ctx, d);
    for (int i = 0; i < n; ++i) {
        leaf2[i] = h[i];
        max2[i] = h[n + i];
    }
}

void launch_rescale(Tree& t, double c, cudaStream_t s) {
    if (t.n == 0) return;
    k_rescale<<<1024, 256, 0, s>>>(t.coef, (size_t)t.n * t.mra->bsize(), c);
    k_rescale<<<64, 256, 0, s>>>(t.norm2, (size_t)t.n, c * c);
    k_rescale<<<64, 256, 0, s>>>(t.wnorm2, (size_t)t.n, c * c);
    MWB_CUDA(cudaGetLastError());
    count(t.mra->ctx, 3);
}

double launch_dot(Tree& a, Tree& b, cudaStream_t s) {
    if (a.n == 0 || b.n == 0) return 0.0;
    Ctx* ctx = a.mra->ctx;
    if (!ctx->ticket) {
        ctx->ticket = (unsigned*)dalloc(ctx, sizeof(unsigned));
        MWB_CUDA(cudaMemsetAsync(ctx->ticket, 0, sizeof(unsigned), s));
    }
    int blocks = (a.n + kDotGroups - 1) / kDotGroups;
    if (dot_in_turn(a.mra->k)) blocks = std::min(blocks, 8 * ctx->num_sms);
    double* part = (double*)dalloc(ctx, sizeof(double) * kDotGroups * blocks);
    double* res = mailbox(ctx);
    TView av = view(a);
#define L_DOT(KK) \
    k_dot<KK><<<blocks, kDotThreads, 0, s>>>(av, a.n, b.coef, b.hkey, b.hval, b.hcap, part, ctx->ticket, res);
    MWB_DISPATCH_K(a.mra->k, L_DOT)
#undef L_DOT
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    dfree(ctx, part);
    MWB_CUDA(cudaStreamSynchronize(s));
    return *reinterpret_cast<volatile double*>(ctx->mbox);
}

// ||a - b|| of two compressed trees on one world (any grids)
double launch_distance(Tree& a, Tree& b, cudaStream_t s) {
    Ctx* ctx = a.mra->ctx;
    const int nmax = std::max(1, std::max(a.n, b.n));
    double* part = (double*)dalloc(ctx, sizeof(double) * nmax);
    double* d = (double*)dalloc(ctx, sizeof(double) * 2);
    MWB_CUDA(cudaMemsetAsync(d, 0, sizeof(double) * 2, s));
    TView av = view(a), bv = view(b);
    if (a.n > 0) {
#define L_DIFF(KK) k_diff_nodes<KK><<<(a.n * 32 + 255) / 256, 256, 0, s>>>(av, a.n, b.coef, b.hkey, b.hval, b.hcap, 0, part);
        MWB_DISPATCH_K(a.mra->k, L_DIFF)
#undef L_DIFF
        k_sum_array<<<1, 1024, 0, s>>>(part, a.n, d);
        count(ctx, 2);
    }
    if (b.n > 0) {
#define L_DIFF(KK) k_diff_nodes<KK><<<(b.n * 32 + 255) / 256, 256, 0, s>>>(bv, b.n, a.coef, a.hkey, a.hval, a.hcap, 1, part);
        MWB_DISPATCH_K(a.mra->k, L_DIFF)
#undef L_DIFF
        k_sum_array<<<1, 1024, 0, s>>>(part, b.n, d + 1);
        count(ctx, 2);
    }
    MWB_CUDA(cudaGetLastError());
    double h[2] = {0.0, 0.0};
    MWB_CUDA(cudaMemcpyAsync(h, d, sizeof(double) * 2, cudaMemcpyDeviceToHost, s));
    MWB_CUDA(cudaStreamSynchronize(s));
    dfree(ctx, part);
    dfree(ctx, d);
    return std::sqrt(h[0] + h[1]);
}

// dst[i] = src[perm[i]] for blocks of bs doubles
__global__ void k_gather_blocks(const double* __restrict__ src, const int* __restrict__ perm, int n, size_t bs,
                                double* __restrict__ dst) {
    const int i = blockIdx.x;
    if (i >= n) return;
    const double* a = src + (size_t)perm[i] * bs;
    double* b = dst + (size_t)i * bs;
    for (size_t e = threadIdx.x; e < bs; e += blockDim.x) b[e] = a[e];
}
void launch_gather_blocks(const double* src, const int* perm, int n, size_t bs, double* dst, cudaStream_t s) {
    if (n <= 0) return;
    k_gather_blocks<<<n, 256, 0, s>>>(src, perm, n, bs, dst);
    MWB_CUDA(cudaGetLastError());
}

// host copies of the key helpers for the driver
uint64_t host_make_key(int depth, long long tx, long long ty, long long tz) { return make_key(depth, tx, ty, tz); }

// the root level of several trees on one world, in two launches: each tree's hash index cleared
// (blockIdx.y = tree), then node i = root key i (Morton order) with no parent, no children and zero
// norms, entered into the index
struct RootTree {
    uint64_t* key;
    int* parent;
    int* child0;
    double* norm2;
    double* wnorm2;
    uint64_t* hkey;
    int* hval;
    uint32_t hcap;
};
__global__ void k_hash_reset_many(const RootTree* __restrict__ ts) {
    const RootTree T = ts[blockIdx.y];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < T.hcap; i += gridDim.x * blockDim.x) {
        T.hkey[i] = kEmptyKey;
        T.hval[i] = -1;
    }
}
__global__ void k_roots_many(const RootTree* __restrict__ ts, const uint64_t* __restrict__ rk, int nroot) {
    const RootTree T = ts[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nroot) return;
    T.key[i] = rk[i];
    T.parent[i] = -1;
    T.child0[i] = -1;
    T.norm2[i] = 0.0;
    T.wnorm2[i] = 0.0;
    hash_insert_one(T.hkey, T.hval, T.hcap, rk[i], i);
}
// every node of several trees into their (cleared) hash indices: blockIdx.y = tree
__global__ void k_hash_insert_many(const RootTree* __restrict__ ts, const int* __restrict__ n) {
    const RootTree T = ts[blockIdx.y];
    const int nn = n[blockIdx.y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
        hash_insert_one(T.hkey, T.hval, T.hcap, T.key[i], i);
}
void trees_rehash(const std::vector<Tree*>& ts) {
    if (ts.empty()) return;
    Ctx* ctx = ts[0]->mra->ctx;
    cudaStream_t s = ctx->stream;
    std::vector<RootTree> rt;
    std::vector<int> n;
    uint32_t maxcap = 0;
    int maxn = 0;
    for (Tree* t : ts) {
        rt.push_back(RootTree{t->key, t->parent, t->child0, t->norm2, t->wnorm2, t->hkey, t->hval, t->hcap});
        n.push_back(t->n);
        maxcap = std::max(maxcap, t->hcap);
        maxn = std::max(maxn, t->n);
    }
    RootTree* d_rt = (RootTree*)dalloc(ctx, sizeof(RootTree) * rt.size());
    int* d_n = (int*)dalloc(ctx, sizeof(int) * n.size());
    upload_bytes(ctx, d_rt, rt.data(), sizeof(RootTree) * rt.size());
    upload_bytes(ctx, d_n, n.data(), sizeof(int) * n.size());
    const unsigned nt = (unsigned)rt.size();
    k_hash_reset_many<<<dim3(std::min<uint32_t>((maxcap + 255) / 256, 1024), nt), 256, 0, s>>>(d_rt);
    if (maxn > 0) k_hash_insert_many<<<dim3(std::min((maxn + 255) / 256, 1024), nt), 256, 0, s>>>(d_rt, d_n);
    MWB_CUDA(cudaGetLastError());
    count(ctx, maxn > 0 ? 2 : 1);
    dfree(ctx, d_rt);
    dfree(ctx, d_n);
}
void trees_make_roots(const std::vector<Tree*>& ts) {
    if (ts.empty()) return;
    const Mra& m = *ts[0]->mra;
    Ctx* ctx = m.ctx;
    cudaStream_t s = ctx->stream;
    std::vector<uint64_t> keys;
    for (int z = 0; z < m.boxes[2]; ++z)
        for (int y = 0; y < m.boxes[1]; ++y)
            for (int x = 0; x < m.boxes[0]; ++x) keys.push_back(host_make_key(0, x, y, z));
    std::sort(keys.begin(), keys.end());
    const int nroot = (int)keys.size();
    std::vector<RootTree> rt;
    uint32_t maxcap = 0;
    for (Tree* t : ts) {
        t->n = 0;
        t->level_begin.clear();
        tree_reserve(*t, nroot);
        rt.push_back(RootTree{t->key, t->parent, t->child0, t->norm2, t->wnorm2, t->hkey, t->hval, t->hcap});
        maxcap = std::max(maxcap, t->hcap);
    }
    UploadPack up(ctx);
    const size_t o_rk = up.add(keys), o_rt = up.add(rt);
    char* d_up = up.send();
    const uint64_t* d_rk = reinterpret_cast<const uint64_t*>(d_up + o_rk);
    const RootTree* d_rt = reinterpret_cast<const RootTree*>(d_up + o_rt);
    const unsigned nt = (unsigned)rt.size();
    k_hash_reset_many<<<dim3(std::min<uint32_t>((maxcap + 255) / 256, 1024), nt), 256, 0, s>>>(d_rt);
    k_roots_many<<<dim3((nroot + 255) / 256, nt), 256, 0, s>>>(d_rt, d_rk, nroot);
    MWB_CUDA(cudaGetLastError());
    count(ctx, 2);
    dfree(ctx, d_up);
    for (Tree* t : ts) {
        t->n = nroot;
        t->level_begin = {0, nroot};
    }
}
void host_key_trans(uint64_t k, long long t[3]) { key_trans(k, t); }

}  // namespace mwb
