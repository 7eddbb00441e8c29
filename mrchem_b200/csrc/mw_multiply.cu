// mw_multiply.cu -- pointwise product of two functions on the device (multiwavelet multiplication)
// and the union-grid helpers it is used with.
//
// Contract: mrcpp::multiply(prec, out, c, a, b[, maxIter]) and mrcpp::build_grid / copy_grid as called
// at reference src/qmfunctions/qmfunction_utils.cpp:209-217 (union grid: build_grid(out, a),
// build_grid(out, b), multiply(..., maxIter = 0); adaptive: multiply on the output's current grid,
// refined until converged), src/qmoperators/two_electron/ExchangePotential.cpp:131,253,312 and
// src/qmfunctions/density_utils.cpp:65-91 (square).
//
// Per output node (scale n): both factors are taken at scale n+1 on the node's 8 children -- the
// reconstructed node block, or, where a factor's tree is coarser, the block generated below its
// deepest existing ancestor (zero wavelets) -- evaluated at the children's k^3 Gauss-Legendre points
// (one (2k)x(2k) matrix per dimension, MV = blkdiag(E, E) F^T), multiplied, and projected back and
// compressed with the projection matrix PF = F blkdiag(W, W) and the scale c 2^{3(n+1)/2}.
// Refinement follows the adaptive projection: after every pass the leaves whose wavelet norm exceeds
// prec ||out|| 2^{-depth/2} are split and their children computed.
//
// Work per node: 9 mode products of a (2k)^3 FP64 tensor on the FP64 matrix instruction (mw_block.cuh); a generated factor
// takes a third of its three instead, after a descent of about as much for the first level and a fifth of that for each
// further one; 2 blocks read and 1 written: bound by the FP64 pipe.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/mwb200.h"
#include "mw_block.cuh"
#include "mw_device.cuh"
#include "mw_umma.cuh"
#include "mw_kernels.cuh"
#include "mw_learned.cuh"

namespace mwb {

void set_last_error(const std::string& msg);

struct MulTree {
    uint64_t* okey;
    double* ocoef;
    double* onorm2;
    double* ownorm2;
    const uint64_t* ahk;
    const int* ahv;
    uint32_t ahcap;
    const double* acoef;
    const uint64_t* bhk;
    const int* bhv;
    uint32_t bhcap;
    const double* bcoef;
    double c;
};

struct MulItem {
    int tree;
    int node;
};

template <int K>
struct MulCfg {
    using B = BX<K, 2 * K>;
    static constexpr size_t SMEM = sizeof(double) * (B::VOL + 4 * B::FRAG + 4 * BX<K, K>::FRAG);
    static constexpr int MINB = K <= 6 ? 4 : K <= 10 ? 2 : 1;
    // the first factor's point values wait in tensor memory: 4 RT doubles per lane and couple of column tiles
    static constexpr int NIT = (B::NZT + 2 * B::NWARP - 1) / (2 * B::NWARP), WORDS = 8 * B::RT;
    static constexpr int TNEED = (B::NWARP + 3) / 4 * NIT * WORDS;
    static constexpr int TCOLS = TNEED <= 32 ? 32 : TNEED <= 64 ? 64 : TNEED <= 128 ? 128 : 256;
    static_assert(TNEED <= 256 && MINB * TCOLS <= 512, "tensor memory");
};

// One output node per block.  Per factor: its block, own or generated below the deepest ancestor (bx_descend: a scaling block
// alone), to the point values in a separable transform; the product goes back through PF.  FP64-bound: 9 mode products per node on
// the matrix instruction (16 us per node and SM at k = 10), two blocks per SM so that one's loads and barriers hide behind
// the other's products.  28 pairs at k = 10: 15.5 ms with a thread per pencil and a whole reconstruction per level of a
// missing node, 5.2 ms now.
template <int K>
__global__ void __launch_bounds__(BX<K, 2 * K>::NTHR, MulCfg<K>::MINB)
    k_mul(const MulItem* __restrict__ items, const MulTree* __restrict__ trees, const double* __restrict__ frMV,
          const double* __restrict__ frPF, const double* __restrict__ frH, int n0) {
    using B = BX<K, 2 * K>;
    using C = MulCfg<K>;
    constexpr int K2 = 2 * K, BS = Geo<K>::BS, RT = B::RT;
    extern __shared__ __align__(16) double msm[];
    __shared__ double red[64];
    __shared__ int found[2][2];
    __shared__ uint32_t tmem_slot;
    double* X = msm;
    double* fq = X + B::VOL;        // MV (A, B order)
    double* fp = fq + 2 * B::FRAG;  // PF (A, B order)
    double* fh = fp + 2 * B::FRAG;  // the half filters' images, for a generated factor
    const MulItem it = items[blockIdx.x];
    const MulTree& T = trees[it.tree];
    const uint64_t key = T.okey[it.node];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, depth = key_depth(key);
    long long tr[3];
    key_trans(key, tr);
    bx_operator(fq, frMV, 2 * B::FRAG, B::NTHR);
    bx_operator(fp, frPF, 2 * B::FRAG, B::NTHR);
    if (warp < 2) {
        int idx, da;
        if (warp == 0) bx_lookup(T.ahk, T.ahv, T.ahcap, key, idx, da);
        else bx_lookup(T.bhk, T.bhv, T.bhcap, key, idx, da);
        if (lane == 0) {
            found[warp][0] = idx;
            found[warp][1] = da;
        }
    }
    if (warp == 2) {
        tmem_alloc(&tmem_slot, C::TCOLS);
        tmem_relinquish();
    }
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t stash = tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * C::NIT * C::WORDS);
    // values of the factors at the children's quadrature points; a square takes its one factor once
    const bool sq = T.acoef == T.bcoef;
    for (int q = sq ? 1 : 0; q < 2; ++q) {
        const int idx = found[q][0], da = found[q][1];
        const double* coef = q ? T.bcoef : T.acoef;
        const bool gen = idx >= 0 && da < depth;
        if (idx >= 0) {
            if (gen) bx_operator(fh, frH, 4 * BX<K, K>::FRAG, B::NTHR);
            bx_load<K, B::NWARP>(X, coef + (size_t)idx * BS);
        } else {  // outside the factor's roots (cannot happen on one world): zero
            for (int e = tid; e < B::VOL; e += B::NTHR) X[e] = 0.0;
        }
        cp_async_wait_all();
        __syncthreads();
        if (gen) {
            bx_descend<K, B::NWARP>(X, fh, tr, depth - da);
            bx_slices<K, K2, K, BX<K, K>::LDO>(X, fq, fq + B::FRAG);
        } else {
            bx_slices<K, K2>(X, fq, fq + B::FRAG);
        }
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < C::NIT; ++i) {
            const int t0 = warp + 2 * B::NWARP * i;
            double v[2][RT][2];
            if (gen) bx_z<K, K2, 2, K>(X, t0, B::NWARP, fq, v);
            else bx_z<K, K2, 2>(X, t0, B::NWARP, fq, v);
            uint32_t w[C::WORDS];
            if (q == 0) {
#pragma unroll
                for (int e = 0; e < 4 * RT; ++e) double_to_words(v[e / (2 * RT)][(e / 2) % RT][e % 2], w[2 * e], w[2 * e + 1]);
                tmem_span_st<0, C::WORDS>(stash + i * C::WORDS, w);
                continue;
            }
            if (!sq) {
                tmem_span_ld<0, C::WORDS>(stash + i * C::WORDS, w);
                tmem_span_wait<0, C::WORDS>(w);
            }
            __syncwarp();  // the columns are read
#pragma unroll
            for (int e = 0; e < 4 * RT; e += 2) {  // the product, in the place of the second factor's columns
                const int h = e / (2 * RT), r = (e / 2) % RT;
                const int c = 8 * r + (lane >> 2), tile = t0 + h * B::NWARP, n = 8 * tile + 2 * (lane & 3);
                const double a0 = sq ? v[h][r][0] : words_to_double(w[2 * e], w[2 * e + 1]);
                const double a1 = sq ? v[h][r][1] : words_to_double(w[2 * e + 2], w[2 * e + 3]);
                if (c < K2 && n < K2 * K2) {
                    double* p = X + c * B::LDP + B::physo(n);
                    p[0] = a0 * v[h][r][0];
                    p[1] = a1 * v[h][r][1];
                }
            }
        }
        tmem_wait_st();
        __syncthreads();
    }
    bx_slices<K, K2>(X, fp, fp + B::FRAG);
    __syncthreads();
    const double fac = T.c * exp2(1.5 * (double)(n0 + depth + 1));
    double* dst = T.ocoef + (size_t)it.node * BS;
    double n2 = 0.0, w2 = 0.0;
    bx_columns<K, K2>(X, fp, [&](int c, int n, double v0, double v1) {
        const int a = n % K2, b = n / K2;
        v0 *= fac;
        v1 *= fac;
        *reinterpret_cast<double2*>(dst + n + K2 * K2 * c) = make_double2(v0, v1);
        n2 += v0 * v0 + v1 * v1;
        const bool sc = b < K && c < K;
        if (!(sc && a < K)) w2 += v0 * v0;
        if (!(sc && a + 1 < K)) w2 += v1 * v1;
    });
    tmem_fence_before_sync();
    block_sum2(n2, w2, red);
    __syncthreads();
    tmem_fence_after_sync();
    if (warp == 2) tmem_dealloc(tmem_slot, C::TCOLS);
    if (tid == 0) {
        T.onorm2[it.node] = n2;
        T.ownorm2[it.node] = w2;
    }
}

// linear combination: one input function of a sum
struct AddIn {
    const uint64_t* hk;
    const int* hv;
    uint32_t hcap;
    const double* coef;
    double c;
};
struct AddOut {
    const uint64_t* key;
    double* coef;
    double* norm2;
    double* wnorm2;
};
constexpr int kAddMaxTerms = 256;

// Block of sum_i c_i f_i at one output node: compressed blocks are linear in the function, so the
// inputs' blocks (own, or generated below the deepest ancestor) are combined as they are.  A lane keeps its
// elements' sums in registers (element pairs in the order of the z product's outputs) and adds an own block
// straight from global memory; a generated one comes from bx_descend.  HBM-bound when the inputs have the
// nodes.
template <int K>
struct AddCfg {
    using B = BX<K, K>;
    static constexpr size_t SMEM = sizeof(double) * (B::VOL + 4 * B::FRAG);
    static constexpr int PAIRS = 4 * K * K * K, PER = (PAIRS + B::NTHR - 1) / B::NTHR;  // element pairs per thread
};
template <int K>
__global__ void __launch_bounds__(BX<K, K>::NTHR, 1)
    k_add(const MulItem* __restrict__ items, AddOut out, const AddIn* __restrict__ in, int nin, const double* __restrict__ frH) {
    using B = BX<K, K>;
    using C = AddCfg<K>;
    constexpr int K2 = 2 * K, BS = Geo<K>::BS;
    extern __shared__ __align__(16) double asm_[];
    __shared__ double red[64];
    __shared__ int found[kAddMaxTerms][2];
    double* X = asm_;
    double* h = X + B::VOL;
    bool filters = false;  // h is loaded
    const int node = items[blockIdx.x].node, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t key = out.key[node];
    const int depth = key_depth(key);
    long long tr[3];
    key_trans(key, tr);
    for (int q = warp; q < nin; q += B::NWARP) {
        int idx, da;
        bx_lookup(in[q].hk, in[q].hv, in[q].hcap, key, idx, da);
        if (lane == 0) {
            found[q][0] = idx;
            found[q][1] = da;
        }
    }
    __syncthreads();
    double acc[C::PER][2];
#pragma unroll
    for (int i = 0; i < C::PER; ++i) acc[i][0] = acc[i][1] = 0.0;
    for (int q = 0; q < nin; ++q) {
        const int idx = found[q][0], da = found[q][1];
        const double cf = in[q].c;
        if (idx < 0) continue;  // outside the function's roots (cannot happen on one world): zero
        const double* blk = in[q].coef + (size_t)idx * BS;
        if (da == depth) {
#pragma unroll
            for (int i = 0; i < C::PER; ++i) {
                const int e = tid + i * B::NTHR;
                if (e < C::PAIRS) {
                    const double2 v = __ldcs(reinterpret_cast<const double2*>(blk) + e);
                    acc[i][0] = fma(cf, v.x, acc[i][0]);
                    acc[i][1] = fma(cf, v.y, acc[i][1]);
                }
            }
            continue;
        }
        __syncthreads();  // X is free
        if (!filters) bx_operator(h, frH, 4 * B::FRAG, B::NTHR);
        filters = true;
        bx_load<K, B::NWARP>(X, blk);
        cp_async_wait_all();
        __syncthreads();
        bx_descend<K, B::NWARP>(X, h, tr, depth - da);
#pragma unroll
        for (int i = 0; i < C::PER; ++i) {
            const int e = tid + i * B::NTHR, a = 2 * (e % K), b = (e / K) % K2, c = e / (K * K2);
            if (e < C::PAIRS && b < K && c < K) {
                const double* p = X + c * B::LDP + B::LDO * b;
                if (a < K) acc[i][0] = fma(cf, p[a], acc[i][0]);
                if (a + 1 < K) acc[i][1] = fma(cf, p[a + 1], acc[i][1]);
            }
        }
    }
    double* dst = out.coef + (size_t)node * BS;
    double n2 = 0.0, w2 = 0.0;
#pragma unroll
    for (int i = 0; i < C::PER; ++i) {
        const int e = tid + i * B::NTHR, a = 2 * (e % K), b = (e / K) % K2, c = e / (K * K2);
        if (e < C::PAIRS) {
            reinterpret_cast<double2*>(dst)[e] = make_double2(acc[i][0], acc[i][1]);
            n2 += acc[i][0] * acc[i][0] + acc[i][1] * acc[i][1];
            const bool sc = b < K && c < K;
            if (!(sc && a < K)) w2 += acc[i][0] * acc[i][0];
            if (!(sc && a + 1 < K)) w2 += acc[i][1] * acc[i][1];
        }
    }
    block_sum2(n2, w2, red);
    if (tid == 0) {
        out.norm2[node] = n2;
        out.wnorm2[node] = w2;
    }
}

#define MWB_MUL_DISPATCH_K(k, F)                                                                \
    switch (k) {                                                                                \
        case 4: F(4); break;                                                                    \
        case 5: F(5); break;                                                                    \
        case 6: F(6); break;                                                                    \
        case 7: F(7); break;                                                                    \
        case 8: F(8); break;                                                                    \
        case 9: F(9); break;                                                                    \
        case 10: F(10); break;                                                                  \
        case 11: F(11); break;                                                                  \
        default: throw Error(MW_ERR_ARG, "multiply supports k = 4..11 (order 3..10)");          \
    }

namespace {

inline double mul_split_threshold(double prec, double ref, int depth) { return prec * ref * std::pow(2.0, -0.5 * depth); }

std::vector<uint64_t> host_keys(Tree& t, cudaStream_t s) {
    std::vector<uint64_t> k(t.n);
    if (t.n > 0) MWB_CUDA(cudaMemcpyAsync(k.data(), t.key, sizeof(uint64_t) * t.n, cudaMemcpyDeviceToHost, s));
    MWB_CUDA(cudaStreamSynchronize(s));
    return k;
}

// Append nodes with the given keys (zero blocks) and restore the level order (parents before
// children, keys ascending); returns the tree's keys in the new order.
std::vector<uint64_t> tree_add_keys(Tree& t, const std::vector<uint64_t>& add, cudaStream_t s) {
    if (!add.empty()) {
        const size_t BS = t.mra->bsize();
        const int n0 = t.n, na = (int)add.size();
        tree_reserve(t, n0 + na);
        MWB_CUDA(cudaMemcpyAsync(t.key + n0, add.data(), sizeof(uint64_t) * na, cudaMemcpyHostToDevice, s));
        MWB_CUDA(cudaMemsetAsync(t.coef + (size_t)n0 * BS, 0, sizeof(double) * BS * na, s));
        MWB_CUDA(cudaMemsetAsync(t.norm2 + n0, 0, sizeof(double) * na, s));
        MWB_CUDA(cudaMemsetAsync(t.wnorm2 + n0, 0, sizeof(double) * na, s));
        MWB_CUDA(cudaStreamSynchronize(s));  // `add` may leave scope
        t.n = n0 + na;
    }
    std::vector<uint64_t> keys = host_keys(t, s);
    trees_rebuild({&t}, {std::vector<char>(t.n, 1)}, {keys});
    std::sort(keys.begin(), keys.end());
    return keys;
}

std::vector<uint64_t> children_keys(uint64_t k) {
    long long tr[3];
    host_key_trans(k, tr);
    const int d = (int)(k >> 59);
    std::vector<uint64_t> c;
    for (int q = 0; q < 8; ++q)
        c.push_back(host_make_key(d + 1, 2 * tr[0] + (q & 1), 2 * tr[1] + ((q >> 1) & 1), 2 * tr[2] + ((q >> 2) & 1)));
    return c;
}

// keys of `inp` that `out` lacks, in order (one block; key order is level order): n[0] = count
__global__ void __launch_bounds__(1024) k_grid_missing(const uint64_t* __restrict__ ikey, int ni, const uint64_t* __restrict__ hk,
                                                       const int* __restrict__ hv, uint32_t hcap, uint64_t* add, int* n) {
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int b = 0; b < ni; b += 1024) {
        const int i = b + threadIdx.x;
        const uint64_t k = i < ni ? ikey[i] : 0;
        const bool f = i < ni && hlookup(hk, hv, hcap, k) < 0;
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (f) add[base + before + __popc(m & ((1u << lane) - 1u))] = k;
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) n[0] = base;
}
struct GridArrays {
    uint64_t* key;
    double* coef;
    double* norm2;
    double* wnorm2;
};
// merge of two key-ordered node lists (the tree's n0 nodes, na new ones with zero blocks) into new arrays: one
// block per node, whose place is its rank in its own list plus its rank in the other
__global__ void __launch_bounds__(256) k_grid_merge(GridArrays old, int n0, const uint64_t* __restrict__ add, int na, size_t bs,
                                                    GridArrays out) {
    const int i = blockIdx.x;
    const bool fresh = i >= n0;
    const uint64_t key = fresh ? add[i - n0] : old.key[i];
    const uint64_t* other = fresh ? old.key : add;
    int lo = 0, hi = fresh ? n0 : na;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (other[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    const size_t at = (size_t)lo + (fresh ? i - n0 : i);
    double2* d = reinterpret_cast<double2*>(out.coef + at * bs);
    const double2* c = reinterpret_cast<const double2*>(old.coef + (size_t)(fresh ? 0 : i) * bs);
    for (size_t e = threadIdx.x; e < bs / 2; e += blockDim.x) d[e] = fresh ? make_double2(0.0, 0.0) : c[e];
    if (threadIdx.x == 0) {
        out.key[at] = key;
        out.norm2[at] = fresh ? 0.0 : old.norm2[i];
        out.wnorm2[at] = fresh ? 0.0 : old.wnorm2[i];
    }
}
// parents and first children from the hash index; the first 32 threads also find the level starts
__global__ void k_grid_link(const uint64_t* __restrict__ key, int n, const uint64_t* __restrict__ hk, const int* __restrict__ hv,
                            uint32_t hcap, int* parent, int* child0, int* level) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 32) {
        const uint64_t first = (uint64_t)i << 59;
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key[mid] < first) lo = mid + 1;
            else hi = mid;
        }
        level[i] = lo;
    }
    if (i >= n) return;
    const uint64_t k = key[i];
    const int d = key_depth(k);
    long long t[3];
    key_trans(k, t);
    parent[i] = d > 0 ? hlookup(hk, hv, hcap, make_key(d - 1, t[0] >> 1, t[1] >> 1, t[2] >> 1)) : -1;
    child0[i] = hlookup(hk, hv, hcap, make_key(d + 1, 2 * t[0], 2 * t[1], 2 * t[2]));
}

// Extend the grid of `out` by the grid of `inp` (both on one world).  On the device, with two read-backs (the number of
// new nodes, the level starts) and one copy of the blocks; sorting and relinking on the host took 0.45 ms per call.
void build_grid(Tree& out, Tree& inp) {
    Ctx* ctx = out.mra->ctx;
    cudaStream_t s = ctx->stream;
    const size_t BS = out.mra->bsize();
    if (out.n == 0) trees_make_roots({&out});
    if (inp.n == 0) return;
    Scratch sc(ctx);
    uint64_t* d_add = sc.get<uint64_t>(inp.n + 1);
    int* d_n = sc.get<int>(33);
    k_grid_missing<<<1, 1024, 0, s>>>(inp.key, inp.n, out.hkey, out.hval, out.hcap, d_add, d_n);
    MWB_CUDA(cudaGetLastError());
    ctx->launches++;
    int na = 0;
    readback(ctx, {{&na, d_n, sizeof(int)}});
    if (na > 0) {
        const int n0 = out.n, n = n0 + na;
        // the merged arrays, with room to grow; they and a larger index are all there before the tree takes them
        // (of a tree that once was larger at most 1 GiB: the old arrays are still there while these are filled)
        const int spare = (int)((size_t)(1 << 30) / (sizeof(double) * BS));
        const int cap = n > out.cap ? std::max(n, 2 * out.cap) : std::min(out.cap, n + spare);
        uint32_t hcap = std::max(out.hcap, 1024u);  // hash index at most half full
        while (hcap < 2u * (uint32_t)n) hcap <<= 1;
        Scratch neu(ctx);
        uint64_t* key = neu.get<uint64_t>(cap);
        int* parent = neu.get<int>(cap);
        int* child0 = neu.get<int>(cap);
        double* coef = neu.get<double>(BS * cap);
        double* norm2 = neu.get<double>(cap);
        double* wnorm2 = neu.get<double>(cap);
        uint64_t* hkey = hcap > out.hcap ? neu.get<uint64_t>(hcap) : nullptr;
        int* hval = hcap > out.hcap ? neu.get<int>(hcap) : nullptr;
        k_grid_merge<<<n, 256, 0, s>>>(GridArrays{out.key, out.coef, out.norm2, out.wnorm2}, n0, d_add, na, BS,
                                       GridArrays{key, coef, norm2, wnorm2});
        MWB_CUDA(cudaGetLastError());
        neu.keep();
        auto take = [&](auto*& old, auto* fresh) {
            dfree(ctx, old);
            old = fresh;
        };
        take(out.key, key);
        take(out.parent, parent);
        take(out.child0, child0);
        take(out.coef, coef);
        take(out.norm2, norm2);
        take(out.wnorm2, wnorm2);
        out.cap = cap;
        out.n = n;
        if (hcap > out.hcap) {
            take(out.hkey, hkey);
            take(out.hval, hval);
            out.hcap = hcap;
        }
        launch_hash_reset(out, s);
        launch_hash_insert(out, 0, n, s);
        k_grid_link<<<(n + 255) / 256, 256, 0, s>>>(out.key, n, out.hkey, out.hval, out.hcap, out.parent, out.child0, d_n + 1);
        MWB_CUDA(cudaGetLastError());
        ctx->launches += 2;
        int level[32];
        readback(ctx, {{level, d_n + 1, sizeof(level)}});
        out.level_begin.clear();
        for (int d = 0; d < 32 && (d == 0 || level[d] < n); ++d) out.level_begin.push_back(level[d]);
        out.level_begin.push_back(n);
    }
}

// split flags of the last levels of several trees in one launch: item q = (tree, node)
struct SplitTree {
    const double* wnorm2;
    const uint64_t* key;
    double thr;
};
__global__ void k_split_flags_many(const int2* __restrict__ items, int n, const SplitTree* __restrict__ ts,
                                   int depth_limit, int* flags) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int2 it = items[q];
    const SplitTree T = ts[it.x];
    flags[q] = (key_depth(T.key[it.y]) < depth_limit && sqrt(T.wnorm2[it.y]) > T.thr) ? 1 : 0;
}

// Refinement passes shared by the product and the linear combination: every pass computes the work
// nodes of all output trees with one launch (`launch(items, d_items)`), then, unless prec <= 0 or the
// pass limit is reached, splits the computed nodes whose wavelet norm exceeds prec ||out|| 2^{-depth/2}
// and makes their children the next work.  Finally every tree is compressed bottom-up with its norms.
template <typename LaunchF>
void refine_passes(double prec, int n, Tree** out, int max_iter, LaunchF&& launch) {
    const Mra* m = out[0]->mra;
    Ctx* ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    // work: the current leaves of every output tree (roots for an empty tree)
    std::vector<std::vector<int>> work(n);
    std::vector<std::vector<uint64_t>> keys(n);
    std::vector<Tree*> empty;
    for (int i = 0; i < n; ++i)
        if (out[i]->n == 0) empty.push_back(out[i]);
    trees_make_roots(empty);  // all empty trees at once; their work is every root (host keys on demand)
    for (int i = 0; i < n; ++i) {
        if (std::find(empty.begin(), empty.end(), out[i]) != empty.end()) {
            for (int q = 0; q < out[i]->n; ++q) work[i].push_back(q);
            continue;
        }
        std::vector<int> c0(out[i]->n);
        MWB_CUDA(cudaMemcpyAsync(c0.data(), out[i]->child0, sizeof(int) * out[i]->n, cudaMemcpyDeviceToHost, s));
        MWB_CUDA(cudaStreamSynchronize(s));
        for (int q = 0; q < out[i]->n; ++q)
            if (c0[q] < 0) work[i].push_back(q);
        keys[i] = host_keys(*out[i], s);
    }
    for (int iter = 0;; ++iter) {
        std::vector<MulItem> items;
        size_t nwork = 0;
        for (int i = 0; i < n; ++i) nwork += work[i].size();
        items.reserve(nwork);  // (lists of 10^4 to 10^5 nodes: their growth showed in a pass)
        for (int i = 0; i < n; ++i)
            for (int q : work[i]) items.push_back({i, q});
        if (items.empty()) break;
        MulItem* d_items = (MulItem*)dalloc(ctx, sizeof(MulItem) * items.size());
        upload_bytes(ctx, s, d_items, items.data(), sizeof(MulItem) * items.size());
        launch(items, d_items);
        MWB_CUDA(cudaGetLastError());
        ctx->launches++;
        dfree(ctx, d_items);
        if (prec <= 0.0 || (max_iter >= 0 && iter >= max_iter)) break;
        std::vector<Tree*> ts(out, out + n);
        std::vector<double> leaf2, max2;
        reduce_norms_many(ts, leaf2, max2, s);
        bool any = false;
        // trees whose work is the whole last level (always so when a tree grows from the roots): split
        // flags of all of them in one launch and one read-back, children appended as the next level
        std::vector<int> full;
        for (int i = 0; i < n; ++i) {
            const Tree& o = *out[i];
            if (work[i].empty()) continue;
            const int L = o.levels();
            const int lb = o.level_begin[L - 1], le = o.level_begin[L];
            if ((int)work[i].size() == le - lb && work[i].front() == lb && work[i].back() == le - 1) full.push_back(i);
        }
        if (!full.empty()) {
            std::vector<int2> its;
            its.reserve(nwork);
            std::vector<SplitTree> st(n, SplitTree{nullptr, nullptr, 0.0});
            for (int i : full) {
                Tree& o = *out[i];
                const int L = o.levels();
                st[i] = SplitTree{o.wnorm2, o.key, mul_split_threshold(prec, std::sqrt(leaf2[i]), L - 1)};
                for (int q = o.level_begin[L - 1]; q < o.level_begin[L]; ++q) its.push_back(int2{i, q});
            }
            const int ni = (int)its.size();
            int2* d_its = (int2*)dalloc(ctx, sizeof(int2) * ni);
            SplitTree* d_st = (SplitTree*)dalloc(ctx, sizeof(SplitTree) * n);
            int* d_flags = (int*)dalloc(ctx, sizeof(int) * ni);
            upload_bytes(ctx, s, d_its, its.data(), sizeof(int2) * ni);
            upload_bytes(ctx, s, d_st, st.data(), sizeof(SplitTree) * n);
            k_split_flags_many<<<(ni + 255) / 256, 256, 0, s>>>(d_its, ni, d_st, m->depth_limit, d_flags);
            MWB_CUDA(cudaGetLastError());
            ctx->launches++;
            std::vector<int> flags(ni);
            readback(ctx, s, {{flags.data(), d_flags, sizeof(int) * ni}});
            dfree(ctx, d_its);
            dfree(ctx, d_st);
            dfree(ctx, d_flags);
            std::vector<Tree*> grow;
            std::vector<std::vector<int>> lists;
            std::vector<int> gi;
            size_t q = 0;
            for (int i : full) {  // items are grouped by tree in `full` order
                std::vector<int> l;
                for (; q < its.size() && its[q].x == i; ++q)
                    if (flags[q]) l.push_back(its[q].y);
                work[i].clear();
                if (l.empty()) continue;
                grow.push_back(out[i]);
                lists.push_back(std::move(l));
                gi.push_back(i);
            }
            std::vector<int> before(gi.size());
            for (size_t g = 0; g < gi.size(); ++g) before[g] = out[gi[g]]->n;
            trees_add_children(grow, lists, s);
            for (size_t g = 0; g < gi.size(); ++g) {
                const int i = gi[g];
                any = true;
                work[i].resize(out[i]->n - before[g]);
                std::iota(work[i].begin(), work[i].end(), before[g]);
                keys[i].clear();  // host keys are refreshed when the general path needs them
            }
        }
        for (int i = 0; i < n; ++i) {
            Tree& o = *out[i];
            if (work[i].empty() || std::find(full.begin(), full.end(), i) != full.end()) continue;
            if (keys[i].size() != (size_t)o.n) keys[i] = host_keys(o, s);
            std::vector<double> w2(o.n);
            MWB_CUDA(cudaMemcpyAsync(w2.data(), o.wnorm2, sizeof(double) * o.n, cudaMemcpyDeviceToHost, s));
            MWB_CUDA(cudaStreamSynchronize(s));
            const double ref = std::sqrt(leaf2[i]);
            std::vector<uint64_t> add;
            for (int q : work[i]) {
                const int d = (int)(keys[i][q] >> 59);
                if (d < m->depth_limit && std::sqrt(w2[q]) > mul_split_threshold(prec, ref, d)) {
                    const std::vector<uint64_t> ch = children_keys(keys[i][q]);
                    add.insert(add.end(), ch.begin(), ch.end());
                }
            }
            work[i].clear();
            if (add.empty()) continue;
            any = true;
            keys[i] = tree_add_keys(o, add, s);
            std::sort(add.begin(), add.end());
            for (uint64_t k : add)
                work[i].push_back((int)(std::lower_bound(keys[i].begin(), keys[i].end(), k) - keys[i].begin()));
        }
        if (!any) break;
    }
    trees_finish(std::vector<Tree*>(out, out + n), false, s);
    MWB_CUDA(cudaStreamSynchronize(s));
}

// out[i] = c[i] a[i] b[i], lock-step passes over the batch
void multiply_batched(double prec, int n, Tree** out, const double* c, Tree** a, Tree** b, int max_iter) {
    const Mra* m = a[0]->mra;
    Ctx* ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    const int K = m->k;
    for (int i = 0; i < n; ++i) {
        if (!out[i] || !a[i] || !b[i]) throw Error(MW_ERR_ARG, "null tree");
        if (out[i]->mra != m || a[i]->mra != m || b[i]->mra != m) throw Error(MW_ERR_ARG, "trees on different worlds");
        if (a[i]->n == 0 || b[i]->n == 0) throw Error(MW_ERR_STATE, "empty input tree");
        for (int j = 0; j < n; ++j)
            if (j != i && out[j] == out[i]) throw Error(MW_ERR_ARG, "output tree listed twice");
        if (out[i] == a[i] || out[i] == b[i]) throw Error(MW_ERR_ARG, "output tree is also an input");
    }
    std::vector<MulTree> mt(n);
    MulTree* d_trees = (MulTree*)dalloc(ctx, sizeof(MulTree) * n);
    refine_passes(prec, n, out, max_iter, [&](const std::vector<MulItem>& items, const MulItem* d_items) {
        for (int i = 0; i < n; ++i) {  // output arrays may have moved (growth) since the last pass
            Tree& o = *out[i];
            mt[i] = MulTree{o.key, o.coef, o.norm2, o.wnorm2, a[i]->hkey, a[i]->hval, a[i]->hcap, a[i]->coef,
                            b[i]->hkey, b[i]->hval, b[i]->hcap, b[i]->coef, c ? c[i] : 1.0};
        }
        MWB_CUDA(cudaMemcpyAsync(d_trees, mt.data(), sizeof(MulTree) * n, cudaMemcpyHostToDevice, s));
#define L_MUL(KK)                                                                                                 \
    {                                                                                                             \
        const size_t smem = MulCfg<KK>::SMEM;                                                                     \
        MWB_CUDA(cudaFuncSetAttribute(k_mul<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));        \
        k_mul<KK><<<(unsigned)items.size(), BX<KK, 2 * KK>::NTHR, smem, s>>>(d_items, d_trees, m->d_frMV, m->d_frPF, \
                                                                             m->d_frH, m->n0);                    \
    }
        MWB_MUL_DISPATCH_K(K, L_MUL)
#undef L_MUL
    });
    dfree(ctx, d_trees);
    MWB_CUDA(cudaStreamSynchronize(s));
}

// out = sum_i c[i] f[i] on one world
void add_trees(double prec, Tree* out, int n, const double* c, Tree** f, int max_iter) {
    if (!out || n <= 0 || !f || !c) throw Error(MW_ERR_ARG, "null tree or empty sum");
    if (n > kAddMaxTerms) throw Error(MW_ERR_ARG, "at most 256 functions per sum");
    const Mra* m = out->mra;
    Ctx* ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    std::vector<AddIn> in(n);
    for (int i = 0; i < n; ++i) {
        if (!f[i]) throw Error(MW_ERR_ARG, "null tree");
        if (f[i]->mra != m) throw Error(MW_ERR_ARG, "trees on different worlds");
        if (f[i]->n == 0) throw Error(MW_ERR_STATE, "empty input tree");
        if (f[i] == out) throw Error(MW_ERR_ARG, "output tree is also an input");
        in[i] = AddIn{f[i]->hkey, f[i]->hval, f[i]->hcap, f[i]->coef, c[i]};
    }
    AddIn* d_in = (AddIn*)dalloc(ctx, sizeof(AddIn) * n);
    MWB_CUDA(cudaMemcpyAsync(d_in, in.data(), sizeof(AddIn) * n, cudaMemcpyHostToDevice, s));
    const int K = m->k;
    Tree* outs[1] = {out};
    refine_passes(prec, 1, outs, max_iter, [&](const std::vector<MulItem>& items, const MulItem* d_items) {
        const AddOut ao{out->key, out->coef, out->norm2, out->wnorm2};
#define L_ADD(KK)                                                                                                   \
    {                                                                                                               \
        const size_t smem = AddCfg<KK>::SMEM;                                                                       \
        MWB_CUDA(cudaFuncSetAttribute(k_add<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));          \
        k_add<KK><<<(unsigned)items.size(), BX<KK, KK>::NTHR, smem, s>>>(d_items, ao, d_in, n, m->d_frH);           \
    }
        MWB_MUL_DISPATCH_K(K, L_ADD)
#undef L_ADD
    });
    dfree(ctx, d_in);
    MWB_CUDA(cudaStreamSynchronize(s));
}

}  // namespace
}  // namespace mwb

struct mw_tree_s : mwb::Tree {};

#define MWM_TRY(...)                                \
    try {                                           \
        __VA_ARGS__;                                \
        return MW_OK;                               \
    } catch (const mwb::Error& e) {                 \
        mwb::set_last_error(e.what());              \
        return e.code;                              \
    } catch (const std::exception& e) {             \
        mwb::set_last_error(e.what());              \
        return MW_ERR_STATE;                        \
    }
#define MWM_ARG(cond, msg) \
    if (!(cond)) throw mwb::Error(MW_ERR_ARG, msg)

extern "C" {

int mw_multiply(double prec, mw_tree out, double c, mw_tree a, mw_tree b, int max_iter) {
    MWM_TRY({
        MWM_ARG(out && a && b, "null tree");
        MWB_CUDA(cudaSetDevice(a->mra->ctx->device));
        mwb::Tree* o = out;
        mwb::Tree* pa = a;
        mwb::Tree* pb = b;
        mwb::multiply_batched(prec, 1, &o, &c, &pa, &pb, max_iter);
    })
}

int mw_multiply_batched(int n, double prec, mw_tree* out, const double* c, mw_tree* a, mw_tree* b, int max_iter) {
    MWM_TRY({
        MWM_ARG(n > 0 && out && a && b, "null pointer or empty batch");
        MWM_ARG(a[0], "null input tree");
        MWB_CUDA(cudaSetDevice(a[0]->mra->ctx->device));
        std::vector<mwb::Tree*> o(n), pa(n), pb(n);
        for (int q = 0; q < n; ++q) {
            o[q] = out[q];
            pa[q] = a[q];
            pb[q] = b[q];
        }
        mwb::multiply_batched(prec, n, o.data(), c, pa.data(), pb.data(), max_iter);
    })
}

int mw_square(double prec, mw_tree out, mw_tree a, int max_iter) { return mw_multiply(prec, out, 1.0, a, a, max_iter); }

int mw_add(double prec, mw_tree out, int n, const double* c, mw_tree* f, int max_iter) {
    MWM_TRY({
        MWM_ARG(out && f && c && n > 0, "null pointer or empty sum");
        MWB_CUDA(cudaSetDevice(out->mra->ctx->device));
        std::vector<mwb::Tree*> v(n);
        for (int q = 0; q < n; ++q) v[q] = f[q];
        mwb::add_trees(prec, out, n, c, v.data(), max_iter);
    })
}

int mw_tree_build_grid(mw_tree out, mw_tree inp) {
    MWM_TRY({
        MWM_ARG(out && inp, "null tree");
        MWM_ARG(out->mra == inp->mra, "trees on different worlds");
        MWM_ARG(out != inp, "a tree cannot extend itself");
        MWB_CUDA(cudaSetDevice(inp->mra->ctx->device));
        mwb::build_grid(*out, *inp);
    })
}

int mw_tree_clear(mw_tree t) {
    MWM_TRY({
        MWM_ARG(t, "null tree");
        t->n = 0;
        t->level_begin.clear();
        if (t->hcap > 0) mwb::launch_hash_reset(*t, t->mra->ctx->stream);
        MWB_CUDA(cudaStreamSynchronize(t->mra->ctx->stream));
    })
}

int mw_tree_copy_grid(mw_tree out, mw_tree inp) {
    const int st = mw_tree_clear(out);
    return st != MW_OK ? st : mw_tree_build_grid(out, inp);
}

}  // extern "C"
