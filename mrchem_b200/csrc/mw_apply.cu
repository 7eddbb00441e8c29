// mw_apply.cu -- batched, adaptive NS-form apply on the device.
//
// A batch is any number of (output tree, operator, input tree) triples sharing one world (e.g. 32
// orbitals with 32 Helmholtz operators).  The refinement passes run in lock-step over the batch:
// pass d handles the depth-d output nodes of every tree with one launch per stage:
//   1. candidates: a block of four warps per output node walks its operator's offset list, looks the input
//      node up in the input tree's hash index (or its leaf ancestor -> generated node) and screens it;
//   2. generated (scaling-only) input nodes are de-duplicated per tree and built once;
//   3. per candidate, the number of terms that pass the screening (the triples it contributes);
//   4. line-ordered engines (FP64, FP32, BF16x3): the triples are expanded and sorted per output node by (term, dz, dy), and
//      each node's sorted triples are cut at plane boundaries into chunks of about chunk_triples
//      triples (a per-engine context setting, 48 unless tuned); the input blocks of the pass get
//      images in the kernel's staging layout.  TF32 and pencil engines: each node's candidate
//      list is cut into chunks of at most chunk_triples triples;
//   5. the contraction kernel runs one CTA per chunk; multi-chunk nodes write partial blocks that
//      a reduction kernel adds in chunk order (deterministic), single-chunk nodes write directly;
//   6. norms and split flags; children are appended to each tree.
// At small sizes a pass is bound by its launches, transfers and allocations, not by the contraction: what the
// host sends goes in one transfer, the counters are cleared by one memset, per-item arrays share one allocation,
// and chunk and partial-slot counts travel packed through one scan (a Poisson apply at order 5, seven passes:
// 2.11 -> 1.69 ms; at order 7: 4.35 -> 4.12 ms).
// Results are identical to the per-node sequential order up to FP64 rounding.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <string>
#include <type_traits>

#include "mw_block.cuh"
#include "mw_device.cuh"
#include "mw_kernels.cuh"
#include "mw_tmem.cuh"
#include "mw_umma.cuh"

namespace mwb {

constexpr double kTensorCoreMinPrec = 1e-6;  // finest prec served by the split-TF32 engine

struct BTree {
    const uint64_t* okey;
    double* ocoef;
    double* onorm2;
    double* ownorm2;
    InView in;
    const uint64_t* inkey;
    const DeltaRec* deltas;
    const TermRec* terms;
    const double* mats;
    const float* mats32;
    const double* matsD;      // fragment images (FP64 matrix-instruction contraction)
    const double* matsE;
    const float* matsT32;     // transposed, zero-padded copies (GEMM-tiled FP32 contraction)
    const float* matsbT32;
    const float* matsI;  // split-TF32 operator images (tensor-core contraction)
    const float* matsbI;
    const float* matsS32;  // tensor-core x step engine: split-layout y/z operators and x-operator slices
    const float* matsbS32;
    const unsigned char* matsX;
    int nprefix;
    int root;
    double theta;
    double thr;  // split threshold of this pass
    int depth;   // depth of this entry's output nodes
    int depth_limit;
    long long ext[3];
    // block images of the pass (line-ordered contraction): input node i of this entry's depth has
    // image slot img_base + i - img_lb, for i in [img_lb, img_le)
    long long img_base;
    int img_lb, img_le;
};

struct Item {
    int tree;
    int node;
};

struct Chunk {
    int item;
    int c0, c1;
    int slot;  // partial block slot, -1: write the output node directly
};

// ---------------------------------------------------------------------------------------------
// 1. candidates
// ---------------------------------------------------------------------------------------------
// One block of four warps per output node (a warp per node walked the root's 6,859 offsets in 214 dependent steps of hash
// probes, 40 us a launch).  First pass (offs == nullptr): counts; second: the candidates in offset order, with their item.
constexpr int kCandThreads = 128;
__global__ void __launch_bounds__(kCandThreads) k_bcand(const Item* __restrict__ items, const BTree* __restrict__ trees,
                                                        int* count, const int* __restrict__ offs, int* cdelta, int* csrc,
                                                        int* cand_item, uint64_t* greq_key, int* greq_leaf, int* ngreq) {
    __shared__ int ws[2][kCandThreads / 32];
    const int w = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool fill = offs != nullptr;
    const Item it = items[w];
    const BTree& T = trees[it.tree];
    const int depth = T.depth;
    const long long ext[3] = {T.ext[0], T.ext[1], T.ext[2]};
    long long to[3];
    key_trans(T.okey[it.node], to);
    int kept = 0, gens = 0;  // count pass: this warp's; fill pass: candidates of the earlier offsets
    const int base = fill ? offs[w] : 0;
    int par = 0;
    for (int b0 = 0; b0 < T.nprefix; b0 += kCandThreads, par ^= 1) {
        const int e = b0 + threadIdx.x;
        int ok = 0, src = 0, leaf = -1;
        uint64_t gk = kEmptyKey;
        if (e < T.nprefix) {
            const DeltaRec de = T.deltas[e];
            long long ti[3];
            bool inside = true;
            for (int d = 0; d < 3; ++d) {
                ti[d] = to[d] - de.d[d];
                if (ti[d] < 0 || ti[d] >= ext[d]) inside = false;
            }
            if (inside) {
                const uint64_t key = make_key(depth, ti[0], ti[1], ti[2]);
                const int idx = hlookup(T.in.hkey, T.in.hval, T.in.hcap, key);
                if (idx >= 0) {
                    const double nu = sqrt(T.in.norm2[idx]);
                    if (nu > 0.0 && de.maxb * nu >= T.theta) { ok = 1; src = idx; }
                } else {
                    for (int da = depth - 1; da >= 0 && leaf < 0; --da) {
                        const int sh = depth - da;
                        leaf = hlookup(T.in.hkey, T.in.hval, T.in.hcap, make_key(da, ti[0] >> sh, ti[1] >> sh, ti[2] >> sh));
                    }
                    const double nul = leaf >= 0 ? sqrt(T.in.norm2[leaf]) : 0.0;
                    if (nul > 0.0 && de.maxb * nul >= T.theta) {
                        ok = 1;
                        // entry index in place of the depth bits (an entry has one depth): unique
                        gk = ((uint64_t)it.tree << 57) | (key & ((1ull << 57) - 1));
                    }
                }
            }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        if (!fill) {  // the counting pass also counts the generated-node requests
            kept += __popc(bal);
            gens += __popc(__ballot_sync(0xffffffffu, ok && gk != kEmptyKey));
            continue;
        }
        if (lane == 0) ws[par][warp] = __popc(bal);
        __syncthreads();  // (the other half of ws is free again: every warp has passed this barrier's predecessor)
        int before = 0, all = 0;
        for (int q = 0; q < kCandThreads / 32; ++q) {
            if (q < warp) before += ws[par][q];
            all += ws[par][q];
        }
        if (ok) {
            const int pos = base + kept + before + __popc(bal & ((1u << lane) - 1u));
            cdelta[pos] = e;
            cand_item[pos] = w;
            if (gk != kEmptyKey) {
                const int r = atomicAdd(ngreq, 1);
                greq_key[r] = gk;
                greq_leaf[r] = leaf;
                csrc[pos] = -(r + 1);
            } else {
                csrc[pos] = src;
            }
        }
        kept += all;
    }
    if (fill) return;
    if (lane == 0) {
        ws[0][warp] = kept;
        if (gens) atomicAdd(ngreq, gens);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int n = 0;
        for (int q = 0; q < kCandThreads / 32; ++q) n += ws[0][q];
        count[w] = n;
    }
}

__global__ void k_bunique_flags(const uint64_t* __restrict__ k, int n, int* flags) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flags[i] = (i == 0 || k[i] != k[i - 1]) ? 1 : 0;
}
__global__ void k_bunique_scatter(const uint64_t* __restrict__ k, const int* __restrict__ leaf,
                                  const int* __restrict__ flags, const int* __restrict__ pos, int n, uint64_t* uk,
                                  int* ul) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (flags[i]) {
        uk[pos[i]] = k[i];
        ul[pos[i]] = leaf[i];
    }
}
__global__ void k_bresolve_gen(int* csrc, int ncand, const uint64_t* __restrict__ greq_key,
                               const uint64_t* __restrict__ ukey, int nu) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncand) return;
    const int s = csrc[i];
    if (s >= 0) return;
    const uint64_t key = greq_key[-s - 1];
    int lo = 0, hi = nu;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ukey[mid] < key) lo = mid + 1; else hi = mid;
    }
    csrc[i] = -(lo + 1);
}

// ---------------------------------------------------------------------------------------------
// 2. generated input nodes: reconstruct the leaf ancestor, take the child on the path, descend
//    with zero wavelets (s_c = H_c^T s per dimension)
// ---------------------------------------------------------------------------------------------
// One block per node, level by level from the leaf's block on the FP64 matrix instruction (bx_descend).
template <int K>
struct GenCfg {
    using B = BX<K, K>;
    static constexpr size_t SMEM = sizeof(double) * (B::VOL + 4 * B::FRAG);
    static constexpr int MINB = K <= 6 ? 4 : K <= 10 ? 2 : 1;
};
template <int K>
__global__ void __launch_bounds__(BX<K, K>::NTHR, GenCfg<K>::MINB)
    k_bgenerate(const uint64_t* __restrict__ ukey, const int* __restrict__ uleaf, const BTree* __restrict__ trees,
                const double* __restrict__ frH, double* gblk, double* gnorm2) {
    using B = BX<K, K>;
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[64];
    double* X = sm;
    double* h = X + B::VOL;
    const int g = blockIdx.x;
    const uint64_t gkey = ukey[g];
    const BTree& T = trees[(int)(gkey >> 57)];
    const int leaf = uleaf[g];
    long long t[3];
    key_trans(gkey & ((1ull << 57) - 1), t);
    bx_operator(h, frH, 4 * B::FRAG, B::NTHR);
    bx_load<K, B::NWARP>(X, T.in.coef + (size_t)leaf * Geo<K>::BS);
    cp_async_wait_all();
    __syncthreads();
    bx_descend<K, B::NWARP>(X, h, t, T.depth - key_depth(T.inkey[leaf]));
    double n2 = 0.0, dmy = 0.0;
    double* out = gblk + (size_t)g * K * K * K;
    for (int e = threadIdx.x; e < K * K * K; e += B::NTHR) {
        const double v = X[e % (K * K) + B::LDP * (e / (K * K))];
        out[e] = v;
        n2 += v * v;
    }
    block_sum2(n2, dmy, red);
    if (threadIdx.x == 0) gnorm2[g] = n2;
}

// ---------------------------------------------------------------------------------------------
// 3-4. triples per candidate, chunks per output node
// ---------------------------------------------------------------------------------------------
__global__ void k_bterms(const int* __restrict__ cand_item, int ncand, const Item* __restrict__ items,
                         const BTree* __restrict__ trees, const int* __restrict__ cdelta, const int* __restrict__ csrc,
                         const double* __restrict__ gnorm2, int* ntrip) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncand) return;
    const BTree& T = trees[items[cand_item[i]].tree];
    const int src = csrc[i];
    const double nu = src < 0 ? sqrt(gnorm2[-src - 1]) : sqrt(T.in.norm2[src]);
    const DeltaRec de = T.deltas[cdelta[i]];
    int n = 0;
    if (nu > 0.0 && !(de.maxb * nu < T.theta))
        for (int t = de.t0; t < de.t1 && !(T.terms[t].bound * nu < T.theta); ++t) ++n;
    ntrip[i] = n;
}
// greedy cut of each node's candidates into chunks of at most `limit` triples (whole
// candidates; at least one chunk per node so that every output block gets written)
// counts and their prefix sums are packed: chunks in the low word, partial slots (of nodes with several chunks) in the high
__device__ __forceinline__ unsigned long long pack_chunks(int nch) {
    return (unsigned)nch | ((unsigned long long)(nch > 1 ? nch : 0) << 32);
}
__global__ void k_bchunks(const int* __restrict__ offs, int nitems, const int* __restrict__ ntrip, int limit, int fill,
                          unsigned long long* nchunk, const unsigned long long* __restrict__ choff, Chunk* chunks) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= nitems) return;
    const int c0 = offs[w], c1 = offs[w + 1];
    int nch = 0, acc = 0, start = c0;
    const int at = fill ? (int)(uint32_t)choff[w] : 0, slot = fill ? (int)(choff[w] >> 32) : 0;
    const int multi = fill ? ((int)(uint32_t)choff[w + 1] - at > 1) : 0;
    for (int c = c0; c < c1; ++c) {
        const int t = ntrip[c];
        if (acc > 0 && acc + t > limit) {
            if (fill) chunks[at + nch] = Chunk{w, start, c, multi ? slot + nch : -1};
            ++nch;
            acc = 0;
            start = c;
        }
        acc += t;
    }
    if (fill) chunks[at + nch] = Chunk{w, start, c1, multi ? slot + nch : -1};
    ++nch;
    if (!fill) nchunk[w] = pack_chunks(nch);
}
// triples of the line-ordered contraction: candidate c contributes its first ntrip[c] term entries,
// at positions toff[c] ..; key = item << 32 | term << 20 | line rank (dz rank << 10 | dy rank),
// value = candidate << 32 | term entry.  A stable sort by key then groups every output node's
// triples by (term, dz, dy), in candidate order inside a line.
__global__ void k_texpand(const int* __restrict__ offs, const int* __restrict__ cand_item, int ncand, const Item* __restrict__ items,
                          const BTree* __restrict__ trees, const int* __restrict__ cdelta,
                          const int* __restrict__ ntrip, const int* __restrict__ toff,
                          const int* __restrict__ csrc, unsigned long long* key, unsigned long long* val, int* err) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncand) return;
    const int w = cand_item[c];
    const BTree& T = trees[items[w].tree];
    const DeltaRec de = T.deltas[cdelta[c]];
    const int n = ntrip[c], p0 = toff[c];
    const int src = csrc[c];
    if (n > 0 && src >= 0 && (src < T.img_lb || src >= T.img_le)) {  // not a node of this depth's level range
        atomicOr(err, 1);
        return;
    }
    // written mirrored inside the item's range, so that after the stable sort a line's triples come in
    // increasing order of their offset's bound (candidates are listed in decreasing order): the tensor
    // core's FP32 accumulation of a line's x sums rounds toward zero when it adds products of a smaller
    // scale to a larger sum, and adding the small contributions first loses fewer of their bits
    const int T0 = toff[offs[w]], T1 = toff[offs[w + 1]];
    for (int j = 0; j < n; ++j) {
        const int te = de.t0 + j;
        const int q = T0 + T1 - 1 - (p0 + j);
        key[q] = ((unsigned long long)w << 32) | ((unsigned long long)T.terms[te].m << 20) | (unsigned)de.lrank;
        val[q] = ((unsigned long long)c << 32) | (unsigned)te;
    }
}
// greedy cut of each node's sorted triples into chunks of about `limit` triples, at plane
// boundaries (a plane = the triples of one (term, dz); at least one chunk per node).  One warp per
// node: the plane starts of 32 triples at a time come from one ballot, and the cut walks the planes
// in order (a plane's size is known when the next one starts)
__global__ void k_tchunks(const int* __restrict__ offs, const int* __restrict__ toff, int nitems,
                          const unsigned long long* __restrict__ key, int limit, int fill, unsigned long long* nchunk,
                          const unsigned long long* __restrict__ choff, Chunk* chunks) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= nitems) return;  // uniform over the warp
    const int t0 = toff[offs[w]], t1 = toff[offs[w + 1]];
    int nch = 0, acc = 0, start = t0, ps = -1;  // ps: start of the plane being measured
    const int at = fill ? (int)(uint32_t)choff[w] : 0, slot = fill ? (int)(choff[w] >> 32) : 0;
    const int multi = fill ? ((int)(uint32_t)choff[w + 1] - at > 1) : 0;
    auto plane_done = [&](int end) {  // plane [ps, end) is complete: cut before it if it overflows
        const int sz = end - ps;
        if (acc > 0 && acc + sz > limit) {
            if (fill && lane == 0) chunks[at + nch] = Chunk{w, start, ps, multi ? slot + nch : -1};
            ++nch;
            acc = 0;
            start = ps;
        }
        acc += sz;
    };
    for (int b = t0; b < t1; b += 32) {
        const int t = b + lane;
        bool st = false;
        if (t < t1)
            st = t == t0 ||
                 ((uint32_t)(key[t] & 0xffffffffull) >> 10) != ((uint32_t)(key[t - 1] & 0xffffffffull) >> 10);
        unsigned m = __ballot_sync(0xffffffffu, st);
        while (m) {
            const int p = b + __ffs(m) - 1;
            m &= m - 1;
            if (ps >= 0) plane_done(p);
            ps = p;
        }
    }
    if (ps >= 0) plane_done(t1);
    if (fill && lane == 0) chunks[at + nch] = Chunk{w, start, t1, multi ? slot + nch : -1};
    ++nch;
    if (!fill && lane == 0) nchunk[w] = pack_chunks(nch);
}
// FP32 block images for the line-ordered contraction: image row a (a < 2k) holds X[a][b + P c] of the
// node block (P = 2k rounded up to 4; zero where b or c >= 2k), so that a CTA stages a block with
// 16-byte copies.  One CTA per block: read coalesced into shared memory, write the rows coalesced.
// Real nodes: entry e (a tree of the pass) contributes input nodes [lb[e], lb[e] + cnt[e]) at slots
// base[e] ..; generated nodes (k^3 scaling blocks) take slots gbase ...
struct ImgSrc {
    const double* coef;
    long long base;
    int lb, cnt;
};
template <int K>
__global__ void __launch_bounds__(256) k_ximage(const ImgSrc* __restrict__ srcs, int nsrc, const double* __restrict__ gblk,
                                                long long nreal, float* __restrict__ img) {
    constexpr int K2 = 2 * K, KP = (K2 + 3) / 4 * 4, NN = KP * KP, BS = K2 * K2 * K2, KKK = K * K * K;
    extern __shared__ __align__(16) unsigned char smraw[];
    float* blk = reinterpret_cast<float*>(smraw);
    const long long slot = blockIdx.x;
    if (slot < nreal) {
        int lo = 0, hi = nsrc - 1;  // last entry with base <= slot
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (srcs[mid].base <= slot) lo = mid;
            else hi = mid - 1;
        }
        const ImgSrc sr = srcs[lo];
        const double* b = sr.coef + (size_t)(sr.lb + (slot - sr.base)) * BS;
        for (int e = threadIdx.x; e < BS; e += blockDim.x) blk[e] = (float)b[e];
    } else {
        const double* g = gblk + (size_t)(slot - nreal) * KKK;
        for (int e = threadIdx.x; e < BS; e += blockDim.x) {
            const int a = e % K2, bb = (e / K2) % K2, c = e / (K2 * K2);
            blk[e] = (a < K && bb < K && c < K) ? (float)g[a + K * (bb + K * c)] : 0.0f;
        }
    }
    __syncthreads();
    float* out = img + (size_t)slot * K2 * NN;
    for (int e = threadIdx.x; e < K2 * NN; e += blockDim.x) {
        const int a = e / NN, j = e - a * NN, b = j % KP, c = j / KP;
        out[e] = (b < K2 && c < K2) ? blk[a + K2 * (b + K2 * c)] : 0.0f;
    }
}

// ---------------------------------------------------------------------------------------------
// 5. contraction (one CTA per chunk), templated on the product type R:
//    R = double: the plain FP64 apply; R = float: FP32 products with FP64 accumulation of every
//    term's contribution (the mixed path).  Per term, three in-place pencil transforms:
//      out += beta (NS_z (x) NS_y (x) NS_x) in       out_sss -= beta (T_z (x) T_y (x) T_x) in_sss
//    (the second only at depth > 0: the s->s block belongs to coarser scales).
//    Each thread owns two pencils per step, so every operator element read from shared memory (as a
//    16-byte vector) feeds two FMA chains; the per-term matrices are double-buffered.
// ---------------------------------------------------------------------------------------------
template <typename R> struct VecT;
template <> struct VecT<double> { using T = double2; static constexpr int V = 2; };
template <> struct VecT<float> { using T = float4; static constexpr int V = 4; };

template <int K, typename R>
struct ACfg {
    static constexpr int K2 = 2 * K;
    static constexpr int NP = K2 * K2;
    static constexpr int LDM = (K2 + 3) / 4 * 4;          // padded operator row (16-byte vectors)
    static constexpr int MS = K2 * LDM;                     // one operator matrix
    static constexpr int P = K2 + 1;
    static constexpr int VOL = P * K2 * K2;                 // padded (2k)^3 tensor
    static constexpr bool STAGE = sizeof(R) * 2 * (size_t)VOL + sizeof(R) * 6 * MS <= 200 * 1024;
    static constexpr int XS = STAGE ? VOL : K * K * K;
    static constexpr int US = K * K * K;
    static constexpr int NT = ((NP / 2) + 31) / 32 * 32;    // two z-pencils per thread
    static constexpr size_t SMEM = sizeof(R) * (size_t)(XS + VOL + 6 * MS + US) + 64 * sizeof(double) + 64;
    __device__ static inline int at(int a, int b, int c) { return a + P * (b + K2 * c); }
};

// round n up to the vector width
template <typename R> __host__ __device__ constexpr int vround(int n) { return (n + VecT<R>::V - 1) / VecT<R>::V * VecT<R>::V; }

// out0[o] = sum_i M[o][i] x0[i], out1[o] = sum_i M[o][i] x1[i] for o < NOUT, i < NIN (x padded with
// zeros up to a multiple of the vector width)
template <typename R, int NIN, int LDM>
__device__ __forceinline__ void dot2(const R* __restrict__ Mrow, const R (&x0)[vround<R>(NIN)],
                                     const R (&x1)[vround<R>(NIN)], R& s0, R& s1) {
    using V = VecT<R>;
    s0 = R(0);
    s1 = R(0);
#pragma unroll
    for (int i = 0; i < vround<R>(NIN); i += V::V) {
        const typename V::T m = *reinterpret_cast<const typename V::T*>(Mrow + i);
        if constexpr (V::V == 2) {
            s0 = fma(m.x, x0[i], s0); s1 = fma(m.x, x1[i], s1);
            s0 = fma(m.y, x0[i + 1], s0); s1 = fma(m.y, x1[i + 1], s1);
        } else {
            s0 = fmaf(m.x, x0[i], s0); s1 = fmaf(m.x, x1[i], s1);
            s0 = fmaf(m.y, x0[i + 1], s0); s1 = fmaf(m.y, x1[i + 1], s1);
            s0 = fmaf(m.z, x0[i + 2], s0); s1 = fmaf(m.z, x1[i + 2], s1);
            s0 = fmaf(m.w, x0[i + 3], s0); s1 = fmaf(m.w, x1[i + 3], s1);
        }
    }
}

// generic pencil step over a padded shared tensor: for the pencils q of the step (two per
// thread iteration), y[o] = sum_i M[o][i] x[i], i < NIN, o < NOUT, in place (pencils are owned).
// base(q) / stride describe where a pencil lives.
template <int K, typename R, int NIN, int NOUT, int NPEN, typename BaseF>
__device__ __forceinline__ void pencil_step(const R* __restrict__ M, R* A, int stride, BaseF base) {
    using C = ACfg<K, R>;
    constexpr int NV = vround<R>(NIN);
    for (int q = 2 * threadIdx.x; q < NPEN; q += 2 * blockDim.x) {
        const bool two = q + 1 < NPEN;
        const int b0 = base(q), b1 = two ? base(q + 1) : b0;
        R x0[NV], x1[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            x0[i] = i < NIN ? A[b0 + i * stride] : R(0);
            x1[i] = i < NIN ? A[b1 + i * stride] : R(0);
        }
#pragma unroll 2
        for (int o = 0; o < NOUT; ++o) {
            R s0, s1;
            dot2<R, NIN, C::LDM>(M + o * C::LDM, x0, x1, s0, s1);
            A[b0 + o * stride] = s0;
            if (two) A[b1 + o * stride] = s1;
        }
    }
}

template <int K, typename R, bool GEN>
__device__ __forceinline__ void chain_xy(const R* Mx, const R* My, R* X, R* T, R* U, bool root, const double* blk,
                                         bool xfrom_global) {
    using C = ACfg<K, R>;
    constexpr int K2 = C::K2;
    constexpr int NIN = GEN ? K : K2;
    (void)blk;
    (void)xfrom_global;
    // x: T[:, b, c] = Mx X[:, b, c]   (pencils (b, c); GEN: b, c < k, inputs a < k)
    {
        constexpr int UX = GEN ? K : K2;
        constexpr int NV = vround<R>(NIN);
        for (int q = 2 * threadIdx.x; q < UX * UX; q += 2 * blockDim.x) {
            const bool two = q + 1 < UX * UX;
            const int bq0 = q % UX, cq0 = q / UX, bq1 = (q + 1) % UX, cq1 = (q + 1) / UX;
            R x0[NV], x1[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                if (i < NIN) {
                    if (C::STAGE) {
                        x0[i] = X[C::at(i, bq0, cq0)];
                        x1[i] = two ? X[C::at(i, bq1, cq1)] : R(0);
                    } else if (GEN) {
                        x0[i] = X[i + K * (bq0 + K * cq0)];
                        x1[i] = two ? X[i + K * (bq1 + K * cq1)] : R(0);
                    } else {
                        x0[i] = (R)__ldg(&blk[i + K2 * (bq0 + K2 * cq0)]);
                        x1[i] = two ? (R)__ldg(&blk[i + K2 * (bq1 + K2 * cq1)]) : R(0);
                    }
                } else {
                    x0[i] = R(0);
                    x1[i] = R(0);
                }
            }
#pragma unroll 2
            for (int o = 0; o < K2; ++o) {
                R s0, s1;
                dot2<R, NIN, C::LDM>(Mx + o * C::LDM, x0, x1, s0, s1);
                T[C::at(o, bq0, cq0)] = s0;
                if (two) T[C::at(o, bq1, cq1)] = s1;
            }
        }
        if (!root) {
            constexpr int KV = vround<R>(K);
            for (int q = 2 * threadIdx.x; q < K * K; q += 2 * blockDim.x) {
                const bool two = q + 1 < K * K;
                const int bq0 = q % K, cq0 = q / K, bq1 = (q + 1) % K, cq1 = (q + 1) / K;
                R x0[KV], x1[KV];
#pragma unroll
                for (int i = 0; i < KV; ++i) {
                    if (i < K) {
                        if (C::STAGE) {
                            x0[i] = X[C::at(i, bq0, cq0)];
                            x1[i] = two ? X[C::at(i, bq1, cq1)] : R(0);
                        } else if (GEN) {
                            x0[i] = X[i + K * (bq0 + K * cq0)];
                            x1[i] = two ? X[i + K * (bq1 + K * cq1)] : R(0);
                        } else {
                            x0[i] = (R)__ldg(&blk[i + K2 * (bq0 + K2 * cq0)]);
                            x1[i] = two ? (R)__ldg(&blk[i + K2 * (bq1 + K2 * cq1)]) : R(0);
                        }
                    } else {
                        x0[i] = R(0);
                        x1[i] = R(0);
                    }
                }
#pragma unroll 2
                for (int o = 0; o < K; ++o) {
                    R s0, s1;
                    dot2<R, K, C::LDM>(Mx + o * C::LDM, x0, x1, s0, s1);
                    U[o + K * (bq0 + K * cq0)] = s0;
                    if (two) U[o + K * (bq1 + K * cq1)] = s1;
                }
            }
        }
    }
    __syncthreads();
    // y (in place): pencils (a, c), GEN: planes c < k, inputs b < k
    {
        constexpr int NC = GEN ? K : K2;
        pencil_step<K, R, NIN, K2, K2 * NC>(My, T, C::P, [](int q) { return ACfg<K, R>::at(q % (2 * K), 0, q / (2 * K)); });
        if (!root)
            pencil_step<K, R, K, K, K * K>(My, U, K, [](int q) { return (q % K) + K * K * (q / K); });
    }
}

template <int K, typename R>
__global__ void __launch_bounds__(ACfg<K, R>::NT, 1)
    k_bapply(const Chunk* __restrict__ chunks, const Item* __restrict__ items, const BTree* __restrict__ trees,
             const int* __restrict__ cdelta, const int* __restrict__ csrc, const double* __restrict__ gblk,
             const double* __restrict__ gnorm2, double* partials, unsigned long long* ntrip_out) {
    using C = ACfg<K, R>;
    constexpr int K2 = C::K2;
    constexpr int BS = K2 * K2 * K2;
    extern __shared__ __align__(16) unsigned char smraw[];
    R* X = reinterpret_cast<R*>(smraw);
    R* T = X + C::XS;
    R* Mb = T + C::VOL;  // [2][3][MS]
    R* U = Mb + 6 * C::MS;
    double* red = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(U + C::US) + 15) & ~uintptr_t(15));
    const Chunk ch = chunks[blockIdx.x];
    const Item it = items[ch.item];
    const BTree& TR = trees[it.tree];
    const R* mats = reinterpret_cast<const R*>(sizeof(R) == 8 ? (const void*)TR.mats : (const void*)TR.mats32);
    const bool root = TR.root != 0;
    const double theta = TR.theta;
    const int tid = threadIdx.x;
    double acc[2][K2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int c = 0; c < K2; ++c) acc[j][c] = 0.0;
    // the thread's two z-pencils (a, b)
    const int pz0 = 2 * tid, pz1 = 2 * tid + 1;
    const bool own0 = pz0 < C::NP, own1 = pz1 < C::NP;
    const int za0 = pz0 % K2, zb0 = pz0 / K2, za1 = pz1 % K2, zb1 = pz1 / K2;
    unsigned long long ntrip = 0;
    auto load_mats = [&](int buf, const TermRec& tr) {
        R* dst = Mb + buf * 3 * C::MS;
        for (int i = tid; i < 3 * C::MS; i += blockDim.x) {
            const int w = i / C::MS, r = (i % C::MS) / C::LDM, cc = (i % C::MS) % C::LDM;
            const int mi = w == 0 ? tr.mx : (w == 1 ? tr.my : tr.mz);
            dst[i] = cc < K2 ? mats[(size_t)mi * C::NP + r * K2 + cc] : R(0);
        }
    };
    for (int ci = ch.c0; ci < ch.c1; ++ci) {
        const int src = csrc[ci];
        const bool gen = src < 0;
        const double nu = gen ? sqrt(gnorm2[-src - 1]) : sqrt(TR.in.norm2[src]);
        const DeltaRec de = TR.deltas[cdelta[ci]];
        if (!(nu > 0.0) || de.maxb * nu < theta) continue;
        if (TR.terms[de.t0].bound * nu < theta) continue;
        const double* blk = gen ? gblk + (size_t)(-src - 1) * K * K * K : TR.in.coef + (size_t)src * BS;
        __syncthreads();  // previous candidate's users of X/T/U/M are done
        if (gen) {
            for (int e2 = tid; e2 < K * K * K; e2 += blockDim.x) {
                const int a = e2 % K, b = (e2 / K) % K, c = e2 / (K * K);
                if (C::STAGE) X[C::at(a, b, c)] = (R)blk[e2]; else X[e2] = (R)blk[e2];
            }
        } else if (C::STAGE) {
            for (int e2 = tid; e2 < BS; e2 += blockDim.x) {
                const int a = e2 % K2, b = (e2 / K2) % K2, c = e2 / (K2 * K2);
                X[C::at(a, b, c)] = (R)blk[e2];
            }
        }
        load_mats(0, TR.terms[de.t0]);
        int buf = 0;
        for (int ti = de.t0; ti < de.t1; ++ti) {
            const TermRec tr = TR.terms[ti];
            if (tr.bound * nu < theta) break;
            const R* Mx = Mb + buf * 3 * C::MS;
            const R* My = Mx + C::MS;
            const R* Mz = My + C::MS;
            __syncthreads();  // X, this term's matrices and the previous z-step are complete
            if (gen) chain_xy<K, R, true>(Mx, My, X, T, U, root, blk, !C::STAGE);
            else chain_xy<K, R, false>(Mx, My, X, T, U, root, blk, !C::STAGE);
            __syncthreads();
            // prefetch the next term's matrices into the other buffer while doing z
            if (ti + 1 < de.t1 && !(TR.terms[ti + 1].bound * nu < theta)) load_mats(buf ^ 1, TR.terms[ti + 1]);
            // z: acc[(a, b)][c'] += beta sum_c Mz[c'][c] T[a, b, c]
            {
                constexpr int NIN = K2;
                const int nin = gen ? K : K2;
                constexpr int NV = vround<R>(NIN);
                R x0[NV], x1[NV];
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    x0[i] = (own0 && i < nin) ? T[C::at(za0, zb0, i)] : R(0);
                    x1[i] = (own1 && i < nin) ? T[C::at(za1, zb1, i)] : R(0);
                }
#pragma unroll
                for (int o = 0; o < K2; ++o) {
                    R s0, s1;
                    dot2<R, NIN, C::LDM>(Mz + o * C::LDM, x0, x1, s0, s1);
                    acc[0][o] = fma(tr.beta, (double)s0, acc[0][o]);
                    acc[1][o] = fma(tr.beta, (double)s1, acc[1][o]);
                }
                if (!root) {
                    constexpr int KV = vround<R>(K);
                    const bool u0 = own0 && za0 < K && zb0 < K, u1 = own1 && za1 < K && zb1 < K;
                    if (u0 || u1) {
                        R y0[KV], y1[KV];
#pragma unroll
                        for (int i = 0; i < KV; ++i) {
                            y0[i] = (u0 && i < K) ? U[za0 + K * (zb0 + K * i)] : R(0);
                            y1[i] = (u1 && i < K) ? U[za1 + K * (zb1 + K * i)] : R(0);
                        }
#pragma unroll
                        for (int o = 0; o < K; ++o) {
                            R s0, s1;
                            dot2<R, K, C::LDM>(Mz + o * C::LDM, y0, y1, s0, s1);
                            if (u0) acc[0][o] = fma(-tr.beta, (double)s0, acc[0][o]);
                            if (u1) acc[1][o] = fma(-tr.beta, (double)s1, acc[1][o]);
                        }
                    }
                }
            }
            buf ^= 1;
            ++ntrip;
        }
    }
    double* dst = ch.slot < 0 ? TR.ocoef + (size_t)it.node * BS : partials + (size_t)ch.slot * BS;
    double n2 = 0.0, w2 = 0.0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const bool own = j == 0 ? own0 : own1;
        const int a = j == 0 ? za0 : za1, b = j == 0 ? zb0 : zb1;
        if (own) {
#pragma unroll
            for (int c = 0; c < K2; ++c) {
                const double v = acc[j][c];
                dst[a + K2 * (b + K2 * c)] = v;
                n2 += v * v;
                if (!(a < K && b < K && c < K)) w2 += v * v;
            }
        }
    }
    block_sum2(n2, w2, red);
    if (tid == 0) {
        if (ch.slot < 0) {
            TR.onorm2[it.node] = n2;
            TR.ownorm2[it.node] = w2;
        }
        atomicAdd(ntrip_out, ntrip);
    }
}

// ---------------------------------------------------------------------------------------------
// 5b. GEMM-tiled contraction.  Each mode product of a term is a GEMM C[2k x (2k)^2] = M A with the
//     data operand in shared memory as k-major rows (row = contracted index, columns = the other two
//     indices), and every step writes its result in the row layout the next step reads:
//        X [a][b + P c]  --x-->  T1 [b][a' + P c]  --y-->  T2 [c][a' + P b']  --z-->  acc [c'][a' + P b']
//     (P = 2k rounded up to a multiple of 4, padding zero).  A thread owns MT rows of NH groups of GW
//     consecutive columns, the groups P/NH slices apart; per contracted index it reads MT operator and
//     NT = NH GW data values with 8- and 16-byte loads and issues MT*NT/2 packed FMAs.
//     Two limits bound the tile: a warp is tied to its SM sub-partition, so the tiles have to give all four
//     the same work; and a shared-memory load delivers 128 bytes a clock to the registers of the whole SM,
//     broadcast or not, so a tile costs MT*NT FMA clocks of its sub-partition and 4 (MT + NT) load clocks
//     of the SM.  P = 20: 5 x 10 tiles were 160 threads in 5 warps, two of them on one sub-partition (density
//     potential at order 9: 39.7 ms contracting); 4 x 8 in 8 warps is even but bound by the loads (33.9 ms: loads
//     busy 78 %, FMA pipe 58 % of active clocks); 4 x 16 in 125 of 128 threads 31.7 ms; 10 x 8 in 100 of 128
//     threads 33.2 ms.  P = 12: 4 x 4 in 108 of 128 threads (3 x 6 in 96 before: 1.52 -> 1.38 ms at k = 6);
//     P = 16 and 24 divide evenly at 4 x 8 and 6 x 6 (wider loads: 2.94 -> 2.25 at k = 8, 10.1 -> 8.3 at k = 12).
//     Operators are staged
//     transposed (At[k][o] = M[o][k]); the z step uses the beta-scaled tables.
//     Below the root the s->s block is taken out with three k x k x k GEMMs on the top-left k x k
//     operator blocks (U1, U2, Uc), each thread one column and all or half of the rows; the owners of the z tiles
//     subtract Uc one phase later.
//     Generated inputs (scaling part only) contract over k instead of 2k and skip the column groups that
//     only see their zero wavelet part: the upper half of every thread's groups in the x and y steps.
//     Barriers per term: after x, after y.  Shared-memory hazards across terms are resolved by
//     loading each operator in a phase that the two barriers separate from its readers:
//     Mx(t+1) and Mz(t) during y(t), My(t+1) during z(t).
// ---------------------------------------------------------------------------------------------
template <int K>
struct GCfg {
    static constexpr int K2 = 2 * K;
    static constexpr int KP = (K2 + 3) / 4 * 4;
    static constexpr int NN = KP * KP;
    static constexpr int MT = KP == 8 ? 2 : KP == 24 ? 6 : 4;   // rows of a thread
    static constexpr int GW = KP == 24 ? 6 : 4;                 // columns of a group (within one slice: GW divides P)
    static constexpr int NH = KP == 20 ? 4 : KP == 16 ? 2 : 1;     // groups of a thread
    static constexpr int NT = NH * GW;
    static constexpr int RT = KP / MT;            // row tiles
    static constexpr int NA = KP / GW;            // groups per slice
    static constexpr int NS = KP / NH;            // slices of first groups
    static constexpr int GS = NN / NH;            // column distance of a thread's groups
    static constexpr int NTILE = RT * NA * NS;
    static constexpr int NTHR = (NTILE + 63) / 64 * 64;
    static constexpr int NWARP = NTHR / 32;
    // Row strides: 16-byte rows.  Of the T1 (x-step output) and T2 (y-step output) buffers they are those with the
    // fewest counted shared-memory wavefronts of a CTA's epilogue stores (P = 20: 704 and 960 against 1208 and 1008 unpadded).
    static constexpr int LDX = NN + 4;  // staged by cp.async from the block images
    static constexpr int LD1 = NN + 4;
    static constexpr int LD2 = NN + (KP == 20 ? 4 : 0);
    static constexpr int KK = K * K;
    static constexpr int KKK = K * K * K;
    // correction tiles: one column and all rows (P = 20: k^2 threads are 3 or 4 warps, one per sub-partition) or half of them
    static constexpr int CH = KP == 20 ? 1 : 2;
    static constexpr int RH = CH == 1 ? (K + 1) / 2 * 2 : (K + 3) / 4 * 2;  // rows of a thread, even
    // contracted indices per step of the tile products' loops (loads of a step are in flight together)
    static constexpr int KU = K % 5 == 0 ? 5 : K % 4 == 0 ? 4 : K % 3 == 0 ? 3 : K == 7 ? 7 : 4;
    static constexpr int ND = MT * NT;          // accumulators per thread
    // accumulators in TMEM, 2 columns per double, warps sharing a lane quarter side by side
    static constexpr int TCOLS_NEED = ((NWARP + 3) / 4) * 2 * ND;
    static constexpr int TCOLS = TCOLS_NEED <= 32 ? 32 : TCOLS_NEED <= 64 ? 64 : TCOLS_NEED <= 128 ? 128
                                 : TCOLS_NEED <= 256 ? 256 : 512;
    static constexpr int XBUF = KP * LDX;                        // one staging buffer: X, or T1 at a line's end
    static constexpr int IMG = K2 * NN;                          // block image: rows a < 2k of X, unpadded
    static constexpr size_t SMEM =
        sizeof(float) * (2 * (size_t)XBUF + (size_t)KP * LD2 + 4 * (size_t)KP * KP + 3 * (size_t)KKK) + 64;
    // resident CTAs: what shared memory allows, at most 8 (P = 8), 5 (12: 96 registers a thread), 3 (16: 168), 2 (20: 128)
    static constexpr int SMB = (int)(233472 / (SMEM + 16 + 1024));
    static constexpr int REGB = KP == 8 ? 8 : KP == 12 ? 5 : KP == 16 ? 3 : KP == 20 ? 2 : 1;
    static constexpr int MINB = SMB < 1 ? 1 : SMB < REGB ? SMB : REGB;
    static constexpr bool FITS = SMEM + 16 + 1024 <= 232448 && CH * KK <= NTHR && TCOLS_NEED <= 512 &&
                                 (size_t)KP * LDX * sizeof(float) >= 64 * sizeof(double) && TCOLS * MINB <= 512;
    static_assert(MT % 2 == 0 && GW % 2 == 0 && KP % MT == 0 && KP % GW == 0 && KP % NH == 0, "tiles");
};

// packed FP32 pairs (sm_100 f32x2 arithmetic): two independent round-to-nearest FMAs per instruction,
// bit-identical to two fmaf calls
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b,
                                                        unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// N floats from shared memory by 16-byte (N a multiple of 4: 16-byte aligned) or 8-byte loads
template <int N>
__device__ __forceinline__ void load_row(const float* __restrict__ p, float (&v)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float4 x = *reinterpret_cast<const float4*>(p + i);
            v[i] = x.x, v[i + 1] = x.y, v[i + 2] = x.z, v[i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const float2 x = *reinterpret_cast<const float2*>(p + i);
            v[i] = x.x, v[i + 1] = x.y;
        }
    }
}
template <int N>
__device__ __forceinline__ void store_row(float* __restrict__ p, const float (&v)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) *reinterpret_cast<float2*>(p + i) = make_float2(v[i], v[i + 1]);
    }
}

// FP32 tile with packed accumulators kept across calls: pc[g][i][j] (+)= sum_k At[k lda + i] times the column pair
// B[k ldb + gs g + 2j], B[k ldb + gs g + 2j + 1] of group g < NG, one f32x2 FMA per pair and contracted index
template <int KD, int KU, int NG, int MT, int NH, int NP>
__device__ __forceinline__ void gemm_tile_packed(const float* __restrict__ ap, int lda, const float* __restrict__ bp,
                                                 int ldb, int gs, unsigned long long (&pc)[NH][MT][NP]) {
#pragma unroll KU
    for (int k = 0; k < KD; ++k) {
        float a[MT];
        load_row<MT>(ap, a);
        unsigned long long a2[MT];
#pragma unroll
        for (int i = 0; i < MT; ++i) a2[i] = pack_f32x2(a[i], a[i]);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            float b[2 * NP];
            load_row<2 * NP>(bp + g * gs, b);
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                const unsigned long long b2 = pack_f32x2(b[2 * j], b[2 * j + 1]);
#pragma unroll
                for (int i = 0; i < MT; ++i) pc[g][i][j] = fma_f32x2(a2[i], b2, pc[g][i][j]);
            }
        }
        ap += lda;
        bp += ldb;
    }
}

// one column of a correction product: c[i] = sum_{k<kdim} At[k lda + i] B[k ldb], row pairs packed
// (A16: the rows of At start on 16-byte boundaries, else on 8-byte ones)
template <int KD, int KU, bool A16, int RH>
__device__ __forceinline__ void gemm_column(const float* __restrict__ ap, int lda, const float* __restrict__ bp, int ldb,
                                            float (&c)[RH]) {
    unsigned long long pc[RH / 2];
#pragma unroll
    for (int i = 0; i < RH / 2; ++i) pc[i] = 0ull;
#pragma unroll KU
    for (int k = 0; k < KD; ++k) {
        const float b = *bp;
        const unsigned long long b2 = pack_f32x2(b, b);
        constexpr int R4 = A16 ? RH / 4 * 4 : 0;
#pragma unroll
        for (int i = 0; i < R4; i += 4) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(ap + i);
            pc[i / 2] = fma_f32x2(a.x, b2, pc[i / 2]);
            pc[i / 2 + 1] = fma_f32x2(a.y, b2, pc[i / 2 + 1]);
        }
#pragma unroll
        for (int i = R4; i < RH; i += 2)
            pc[i / 2] = fma_f32x2(*reinterpret_cast<const unsigned long long*>(ap + i), b2, pc[i / 2]);
        ap += lda;
        bp += ldb;
    }
#pragma unroll
    for (int i = 0; i < RH / 2; ++i) unpack_f32x2(pc[i], c[2 * i], c[2 * i + 1]);
}

// Line-ordered GEMM-tiled contraction.  A chunk is a range of one output node's surviving triples,
// sorted by (term, dz, dy): a *line* is a run of triples with the same (term, dz, dy) and a *plane* a
// run with the same (term, dz).  Because a term's operator is separable,
//   sum_l  Mz(dz) My(dy) Mx(dx) in_l  =  sum_dz Mz(dz) [ sum_dy My(dy) [ sum_dx Mx(dx) in_l ] ],
// so every triple costs one x mode product (summed over its line in registers), every line one y mode
// product (summed over its plane in T2) and every plane one z mode product (summed into the output
// block), instead of three mode products per triple.  The s->s correction below the root follows the
// same grouping on its k^3 blocks.
// Input blocks are staged from their images (the X layout in FP32, built per pass) into two buffers
// by cp.async: the next triple's block and operator load while the current triple computes.  At a
// line's end its x sums (T1) replace the line's last block in its buffer.
// tkey (sorted): item << 32 | term << 20 | dz rank << 10 | dy rank; tval: candidate << 32 | term entry.
template <int K>
__global__ void __launch_bounds__(GCfg<K>::NTHR, GCfg<K>::MINB)
    k_gapply(const Chunk* __restrict__ chunks, const Item* __restrict__ items, const BTree* __restrict__ trees,
             const unsigned long long* __restrict__ tkey, const unsigned long long* __restrict__ tval,
             const int* __restrict__ csrc, const float* __restrict__ ximg, long long gbase, double* partials,
             unsigned long long* ntrip_out) {
    using C = GCfg<K>;
    constexpr int K2 = C::K2, KP = C::KP, MT = C::MT, NT = C::NT, GW = C::GW, NH = C::NH, RH = C::RH, KU = C::KU, ND = C::ND;
    constexpr bool A16 = C::CH == 1 || RH % 4 == 0;
    constexpr int LDX = C::LDX, LD1 = C::LD1, LD2 = C::LD2, NN = C::NN, GS = C::GS, IMG = C::IMG;
    constexpr int KK = C::KK, KKK = C::KKK;
    constexpr int BS = K2 * K2 * K2;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ uint32_t tmem_slot;
    float* XA = reinterpret_cast<float*>(smraw);  // staging buffers: X [KP][LDX], or T1 [KP][LD1]
    float* XB = XA + C::XBUF;
    float* T2 = XB + C::XBUF;                 // [KP][LD2]
    float* Mx0 = T2 + KP * LD2;               // [KP][KP], At[k][o] = M[o][k]; x operators of the two buffers
    float* Mx1 = Mx0 + KP * KP;
    float* My = Mx1 + KP * KP;
    float* Mz = My + KP * KP;
    float* U1 = Mz + KP * KP;  // [K][K][K]
    float* U2 = U1 + KKK;
    float* Uc = U2 + KKK;
    const Chunk ch = chunks[blockIdx.x];
    const Item it = items[ch.item];
    const BTree& TR = trees[it.tree];
    const float* mats = TR.matsT32;
    const float* matsb = TR.matsbT32;
    const bool root = TR.root != 0;
    const int tid = threadIdx.x, warp = tid >> 5;
    // tiles: the groups of a slice fastest, then row tiles (fewest wavefronts of the T2 sums), then slices
    const bool own = tid < C::NTILE;
    const int tile = own ? tid : 0;
    const int o0 = (tile / C::NA) % C::RT * MT;
    const int tb0 = tile % C::NA * GW, tc0 = tile / (C::NA * C::RT);  // x tile: first b, c;  y tile: first a', c;
    const int n0 = tb0 + KP * tc0;                                    // z tile: first a', b' (of the first group)
    // correction tile: column n of k^2, rows co0 .. co0 + RH of k (the same rows for a whole warp)
    const int ch0 = tid / (C::NTHR / C::CH), cn = tid - ch0 * (C::NTHR / C::CH);
    const bool cown = !root && cn < KK;
    const int co0 = ch0 * RH, cnl = cown ? cn % K : 0, cnh = cown ? cn / K : 0;

    // accumulators: this thread's TMEM lane
    if (warp == 0) {
        tmem_alloc(&tmem_slot, C::TCOLS);
        tmem_relinquish();
    }
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t tacc = tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * 2 * ND);
    tmem_visit<ND, true>(tacc, [&](int, int n, auto& r) {
#pragma unroll
        for (int q = 0; q < 2 * n; ++q) r[q] = 0u;
    });
    unsigned long long ntrip = 0;
    bool pend2 = false;     // c2 holds a correction block not yet written to Uc
    bool uc_valid = false;  // Uc holds a correction block not yet subtracted
    float c2[RH], u1[RH];   // correction blocks: of the plane, x sums of the line
    unsigned long long xp[NH][MT][GW / 2];  // x sums of the current line (this thread's x tile), column pairs packed

    // asynchronous copy of a transposed operator (At[k][o] = M[o][k], P x P) into shared memory, as
    // one commit group
    auto load_mat = [&](float* dst, const float* tab, int mi) {
        constexpr int NV = KP * KP * (int)sizeof(float) / 16;
        const char* src = reinterpret_cast<const char*>(tab + (size_t)mi * KP * KP);
        for (int e = tid; e < NV; e += blockDim.x) cp_async16(reinterpret_cast<char*>(dst) + 16 * e, src + 16 * e);
        cp_async_commit();
    };
    auto image_of = [&](int t) -> const float* {
        const int src = csrc[(int)(tval[t] >> 32)];
        const long long slot = src < 0 ? gbase + (-src - 1) : TR.img_base + (src - TR.img_lb);
        return ximg + (size_t)slot * IMG;
    };
    // triple t's block image into buffer q (rows a < 2k; the rows of X beyond are never read) and its
    // x operator, one commit group
    auto stage = [&](int t, int q) {
        const float* img = image_of(t);
        float* dst = q ? XB : XA;
        constexpr int RV = NN * (int)sizeof(float) / 16;  // 16-byte vectors per row
        constexpr int EV = 16 / (int)sizeof(float);
        for (int e = tid; e < K2 * RV; e += blockDim.x) {
            const int a = e / RV, v = e - a * RV;
            cp_async16(dst + a * LDX + v * EV, img + (size_t)a * NN + v * EV);
        }
        load_mat(q ? Mx1 : Mx0, mats, TR.terms[(int)(tval[t] & 0xffffffffull)].mx);
    };
    // correction block of element (c', a', b') of this thread's z tile, 0 outside s->s
    auto uc_at = [&](int i, int j) -> double {
        const int cz = o0 + i, ax = tb0 + j % GW, by = tc0 + j / GW * C::NS;
        return (cz < K && ax < K && by < K) ? (double)Uc[cz * KK + ax + K * by] : 0.0;
    };
    auto write_c2 = [&]() {
        if (!cown) return;
#pragma unroll
        for (int i = 0; i < RH; ++i)
            if (co0 + i < K) Uc[(co0 + i) * KK + cn] = c2[i];
    };

    auto line_of = [&](int t) -> uint32_t { return (uint32_t)(tkey[t] & 0xffffffffull); };
    bool line_gen = true;    // every triple of the current line has a generated (scaling-only) input
    bool plane_gen = true;   // ... of the current plane
    bool first_line = true;  // the current line is the first of its plane
    if (ch.c0 < ch.c1) stage(ch.c0, 0);
    int q = 0;  // buffer of the current triple
    for (int t = ch.c0; t < ch.c1; ++t, q ^= 1) {
        const unsigned long long tv = tval[t];
        const bool gen = csrc[(int)(tv >> 32)] < 0;
        const TermRec tr = TR.terms[(int)(tv & 0xffffffffull)];
        const uint32_t lk = line_of(t);
        const bool lstart = t == ch.c0 || line_of(t - 1) != lk;
        const bool pstart = t == ch.c0 || (line_of(t - 1) >> 10) != (lk >> 10);
        const bool lend = t + 1 == ch.c1 || line_of(t + 1) != lk;
        const bool pend = t + 1 == ch.c1 || (line_of(t + 1) >> 10) != (lk >> 10);
        const bool more = t + 1 < ch.c1;
        if (pstart) {
            plane_gen = true;
            first_line = true;
        }
        if (lstart) line_gen = true;
        line_gen = line_gen && gen;
        plane_gen = plane_gen && gen;
        cp_async_wait_all();
        __syncthreads();  // triple t's block and x operator are in; every reader of the other buffer, of
                          // My, Mz, T2, U1, U2 and Uc from earlier steps is done
        if (lend) load_mat(My, mats, tr.my);
        if (pend) load_mat(Mz, matsb, tr.mz);
        if (more) stage(t + 1, q ^ 1);
        if (tid == 0 && t + 2 < ch.c1) prefetch_l2_bulk(image_of(t + 2), (unsigned)(IMG * sizeof(float)));
        float* Xq = q ? XB : XA;
        const float* Mxq = q ? Mx1 : Mx0;
        // ---- x: xp[a'][b + P c] (+)= sum_a Mx[a'][a] X[a][b + P c]   (a line sums its triples)
        if (own) {
            if (lstart) {
#pragma unroll
                for (int g = 0; g < NH; ++g)
#pragma unroll
                    for (int i = 0; i < MT; ++i)
#pragma unroll
                        for (int j = 0; j < GW / 2; ++j) xp[g][i][j] = 0ull;
            }
            // of a generated input, groups outside b, c < k are zero (the upper half of a thread's are: P/2 >= k)
            if (!gen) gemm_tile_packed<K2, KU, NH>(Mxq + o0, KP, Xq + n0, LDX, GS, xp);
            else if (tb0 < K && tc0 < K) gemm_tile_packed<K, KU, (NH + 1) / 2>(Mxq + o0, KP, Xq + n0, LDX, GS, xp);
        }
        if (cown) {  // U1[b][a' + k c] (+)= sum_{a<k} Tx[a'][a] X[a][b + P c]   (summed over the line)
            float c[RH];
            gemm_column<K, KU, A16>(Mxq + co0, KP, Xq + cnl + KP * cnh, LDX, c);
#pragma unroll
            for (int i = 0; i < RH; ++i) u1[i] = lstart ? c[i] : u1[i] + c[i];
        }
        ++ntrip;
        if (!lend) continue;
        __syncthreads();  // every reader of Xq is done: the line's x sums replace its last block
        float* T1 = Xq;       // [KP][LD1]
        if (own) {
#pragma unroll
            for (int g = 0; g < NH; ++g)
#pragma unroll
                for (int j = 0; j < GW / 2; ++j) {
                    float lo[MT], hi[MT];
#pragma unroll
                    for (int i = 0; i < MT; ++i) unpack_f32x2(xp[g][i][j], lo[i], hi[i]);
                    float* col = T1 + (tb0 + 2 * j) * LD1 + o0 + KP * (tc0 + g * C::NS);
                    store_row<MT>(col, lo);
                    store_row<MT>(col + LD1, hi);
                }
        }
        if (cown) {
#pragma unroll
            for (int i = 0; i < RH; ++i)
                if (co0 + i < K) U1[cnl * KK + co0 + i + K * cnh] = u1[i];
        }
        // My (and Mz) were committed before the next triple's staging group
        if (more) cp_async_wait_group<1>();
        else cp_async_wait_all();
        __syncthreads();  // T1, U1, My and Mz are in
        // ---- y: T2[c][a' + P b'] (+)= sum_b My[b'][b] T1[b][a' + P c]   (a plane sums its lines)
        if (pend2) {  // the previous plane's correction block, subtracted in this plane's z phase
            write_c2();
            pend2 = false;
            uc_valid = true;
        }
        if (own) {
            // sums of group g: those of a generated line are zero for c >= k (the upper half of the groups)
            unsigned long long pc[NH][MT][GW / 2];
#pragma unroll
            for (int g = 0; g < NH; ++g)
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int j = 0; j < GW / 2; ++j) pc[g][i][j] = 0ull;
            if (!line_gen) gemm_tile_packed<K2, KU, NH>(My + o0, KP, T1 + n0, LD1, GS, pc);
            else if (tc0 < K) gemm_tile_packed<K, KU, (NH + 1) / 2>(My + o0, KP, T1 + n0, LD1, GS, pc);
#pragma unroll
            for (int g = 0; g < NH; ++g) {
                if (line_gen && !first_line && !(tc0 + g * C::NS < K)) continue;
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    float* row = T2 + (tc0 + g * C::NS) * LD2 + tb0 + KP * (o0 + i);
                    float c[GW], v[GW];
#pragma unroll
                    for (int j = 0; j < GW / 2; ++j) unpack_f32x2(pc[g][i][j], c[2 * j], c[2 * j + 1]);
                    if (!first_line) {
                        load_row<GW>(row, v);
#pragma unroll
                        for (int j = 0; j < GW; ++j) c[j] = v[j] + c[j];
                    }
                    store_row<GW>(row, c);
                }
            }
        }
        if (cown) {  // U2[c][a' + k b'] (+)= sum_{b<k} Ty[b'][b] U1[b][a' + k c]
            float c[RH];
            gemm_column<K, KU, A16>(My + co0, KP, U1 + cn, KK, c);
#pragma unroll
            for (int i = 0; i < RH; ++i)
                if (co0 + i < K) {
                    float& d = U2[cnh * KK + cnl + K * (co0 + i)];
                    d = first_line ? c[i] : d + c[i];
                }
        }
        first_line = false;
        if (!pend) continue;
        __syncthreads();  // T2, U2 and Uc of the plane are complete
        // ---- z: acc[c'][a' + P b'] += sum_c (beta Mz)[c'][c] T2[c][a' + P b']  (- previous correction)
        {
            unsigned long long pc[NH][MT][GW / 2];
#pragma unroll
            for (int g = 0; g < NH; ++g)
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int j = 0; j < GW / 2; ++j) pc[g][i][j] = 0ull;
            if (own) {
                if (plane_gen) gemm_tile_packed<K, KU, NH>(Mz + o0, KP, T2 + n0, LD2, GS, pc);
                else gemm_tile_packed<K2, KU, NH>(Mz + o0, KP, T2 + n0, LD2, GS, pc);
            }
            const bool fold = uc_valid && own;
            tmem_visit<ND, true>(tacc, [&](int d0, int n, auto& r) {
#pragma unroll
                for (int q2 = 0; q2 < n; ++q2) {
                    const int d = d0 + q2, i = d / NT, j = d % NT;
                    float lo, hi;
                    unpack_f32x2(pc[j / GW][i][j % GW / 2], lo, hi);
                    double v = words_to_double(r[2 * q2], r[2 * q2 + 1]) + (double)(j % 2 ? hi : lo);
                    if (fold) v -= uc_at(i, j);
                    double_to_words(v, r[2 * q2], r[2 * q2 + 1]);
                }
            });
        }
        uc_valid = false;
        if (cown) {  // c2[c'][a' + k b'] = sum_{c<k} (beta Tz)[c'][c] U2[c][a' + k b']
            gemm_column<K, KU, A16>(Mz + co0, KP, U2 + cn, KK, c2);
        }
        pend2 = !root;
    }
    cp_async_wait_all();
    __syncthreads();  // z-phase readers of Uc are done
    if (pend2) write_c2();
    uc_valid = pend2;
    __syncthreads();
    double* dst = ch.slot < 0 ? TR.ocoef + (size_t)it.node * BS : partials + (size_t)ch.slot * BS;
    double n2 = 0.0, w2 = 0.0;
    auto emit = [&](int i, int j, double v) {
        const int cz = o0 + i, ax = tb0 + j % GW, by = tc0 + j / GW * C::NS;
        if (uc_valid) v -= uc_at(i, j);
        if (cz < K2 && ax < K2 && by < K2) {
            dst[ax + K2 * (by + K2 * cz)] = v;
            n2 += v * v;
            if (!(ax < K && by < K && cz < K)) w2 += v * v;
        }
    };
    tmem_visit<ND, false>(tacc, [&](int d0, int n, auto& r) {
#pragma unroll
        for (int q = 0; q < n; ++q) {
            const int d = d0 + q;
            if (own) emit(d / NT, d % NT, words_to_double(r[2 * q], r[2 * q + 1]));
        }
    });
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    if (warp == 0) tmem_dealloc(tmem_slot, C::TCOLS);
    double* red = reinterpret_cast<double*>(XA);  // the staging buffers are no longer read
    __syncthreads();
    block_sum2(n2, w2, red);
    if (tid == 0) {
        if (ch.slot < 0) {
            TR.onorm2[it.node] = n2;
            TR.ownorm2[it.node] = w2;
        }
        atomicAdd(ntrip_out, ntrip);
    }
}

}  // namespace mwb
#include "mw_tapply.cuh"
#include "mw_happly.cuh"
#include "mw_dapply.cuh"
namespace mwb {

// triples of every chunk (the sort key of the longest-first launch order); chunks never exceed 2^16 triples
__global__ void k_chunk_len(const Chunk* __restrict__ chunks, int n, int* __restrict__ len) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) len[i] = min(chunks[i].c1 - chunks[i].c0, 65535);
}

// add the partial blocks of a multi-chunk node in chunk order; write block and norms
template <int K>
__global__ void __launch_bounds__(256) k_breduce(const Chunk* __restrict__ chunks, const unsigned long long* __restrict__ choff,
                                                 const Item* __restrict__ items, const BTree* __restrict__ trees,
                                                 const double* __restrict__ partials) {
    using G = Geo<K>;
    __shared__ double red[64];
    const int w = blockIdx.x;
    const int cb = (int)(uint32_t)choff[w], ce = (int)(uint32_t)choff[w + 1];
    if (ce - cb < 2) return;  // a single chunk wrote the node itself
    const Item it = items[w];
    const BTree& TR = trees[it.tree];
    double n2 = 0.0, w2 = 0.0;
    for (int e = threadIdx.x; e < G::BS; e += blockDim.x) {
        double v = 0.0;
        for (int c = cb; c < ce; ++c) v += partials[(size_t)chunks[c].slot * G::BS + e];
        TR.ocoef[(size_t)it.node * G::BS + e] = v;
        const int a = e % G::K2, b = (e / G::K2) % G::K2, cc = e / (G::K2 * G::K2);
        n2 += v * v;
        if (!(a < K && b < K && cc < K)) w2 += v * v;
    }
    block_sum2(n2, w2, red);
    if (threadIdx.x == 0) {
        TR.onorm2[it.node] = n2;
        TR.ownorm2[it.node] = w2;
    }
}

// ---------------------------------------------------------------------------------------------
// 6. per-tree root norms, split flags
// ---------------------------------------------------------------------------------------------
// per entry: the square norm of its nodes, and a root entry's split threshold from it: prec g0 with g0 the root level's
// norm (the same operations as the host's prec g0 2^(-depth/2) at depth 0)
__global__ void k_root_thr(const Item* __restrict__ items, const int* __restrict__ item_off, BTree* trees,
                           const double* __restrict__ prec, double* out) {
    __shared__ double red[64];
    const int t = blockIdx.x;
    double s = 0.0, d = 0.0;
    for (int i = item_off[t] + threadIdx.x; i < item_off[t + 1]; i += blockDim.x) s += trees[t].onorm2[items[i].node];
    block_sum2(s, d, red);
    if (threadIdx.x != 0) return;
    out[t] = s;
    if (trees[t].depth != 0) return;
    const double g0 = sqrt(s);
    trees[t].thr = (prec[t] > 0.0 && g0 > 0.0) ? prec[t] * g0 : INFINITY;
}
__global__ void k_bsplit_flags(const Item* __restrict__ items, int nitems, const BTree* __restrict__ trees,
                               int* flags) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nitems) return;
    const Item it = items[i];
    const BTree& T = trees[it.tree];
    flags[i] = (T.depth < T.depth_limit && sqrt(T.ownorm2[it.node]) > T.thr) ? 1 : 0;
}

// ---------------------------------------------------------------------------------------------
// driver
// ---------------------------------------------------------------------------------------------

static inline void count(Ctx* c, int n = 1) { c->launches += n; }

// MWB200_CONTRACTION=pencil selects the pencil contraction kernel in place of the FP64 and FP32 engines
// (both compute the same sums; kept for comparison)
static bool contraction_pencil() {
    static const bool v = [] {
        const char* e = std::getenv("MWB200_CONTRACTION");
        return e != nullptr && std::string(e) == "pencil";
    }();
    return v;
}

// exclusive sum of d_in[0 .. n) into d_out[0 .. n] (the total lands in d_out[n]; d_in[n] is read, its value is not
// used); no host read-back
template <typename T>
static void scan_only(Ctx* ctx, const T* d_in, T* d_out, int n) {
    size_t tmp = 0;
    MWB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, d_in, d_out, n + 1, ctx->stream));
    void* d_tmp = dalloc(ctx, tmp);
    MWB_CUDA(cub::DeviceScan::ExclusiveSum(d_tmp, tmp, d_in, d_out, n + 1, ctx->stream));
    dfree(ctx, d_tmp);
}
static int scan_total(Ctx* ctx, const int* d_in, int* d_out, int n) {
    size_t tmp = 0;
    MWB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, d_in, d_out, n + 1, ctx->stream));
    void* d_tmp = dalloc(ctx, tmp);
    MWB_CUDA(cub::DeviceScan::ExclusiveSum(d_tmp, tmp, d_in, d_out, n + 1, ctx->stream));
    dfree(ctx, d_tmp);
    int total = 0;
    readback(ctx, {{&total, d_out + n, sizeof(int)}});
    return total;
}

#define MWB_DISPATCH_K(k, F)                                             \
    switch (k) {                                                         \
        case 4: F(4); break;                                             \
        case 5: F(5); break;                                             \
        case 6: F(6); break;                                             \
        case 7: F(7); break;                                             \
        case 8: F(8); break;                                             \
        case 9: F(9); break;                                             \
        case 10: F(10); break;                                           \
        case 11: F(11); break;                                           \
        case 12: F(12); break;                                           \
        default: throw Error(-1, "unsupported order (k must be 4..12)"); \
    }

// launches of the tensor-core x step engine (instantiated only for the orders it serves)
template <int K>
static void* launch_simage(Ctx* ctx, long long nimg, const ImgSrc* d_srcs, int nt, const double* d_gblk,
                           long long nreal, cudaStream_t s) {
    if constexpr (HCfg<K>::FITS) {
        void* img = dalloc(ctx, (size_t)nimg * HCfg<K>::IMGB);
        const long long rows = nimg * (long long)HCfg<K>::R;  // one thread per data row
        k_simage<K><<<(unsigned)((rows + 255) / 256), 256, 0, s>>>(d_srcs, nt, d_gblk, nreal, nimg, (unsigned char*)img);
        return img;
    } else {
        throw Error(-1, "BF16x3 engine: unsupported order");
    }
}
template <int K>
static void launch_happly(int nchunks, const Chunk* d_chunks, const Item* d_items, const BTree* d_trees,
                          const unsigned long long* d_tkey, const unsigned long long* d_tval, const int* d_csrc,
                          const unsigned char* d_img, long long nreal, double* d_partials,
                          unsigned long long* d_ntrip, int* d_kerr, cudaStream_t s) {
    if constexpr (HCfg<K>::FITS) {
        const size_t smem = HCfg<K>::SMEM;
        MWB_CUDA(cudaFuncSetAttribute(k_happly<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_happly<K><<<nchunks, HCfg<K>::NTHR, smem, s>>>(d_chunks, d_items, d_trees, d_tkey, d_tval, d_csrc, d_img,
                                                          nreal, d_partials, d_ntrip, d_kerr);
    } else {
        throw Error(-1, "BF16x3 engine: unsupported order");
    }
}

void run_batch_pass(BatchPass& bp, cudaStream_t s) {
    const int nt = (int)bp.trees.size();
    Ctx* ctx = bp.trees[0].out->mra->ctx;
    const Mra& m = *bp.trees[0].out->mra;
    const int K = m.k;
    const size_t BS = m.bsize();
    // items (output nodes of this depth, grouped by tree) and tree descriptors
    std::vector<Item> items;
    std::vector<int> item_off(nt + 1, 0);
    std::vector<BTree> bt(nt);
    long long nreal = 0;  // block images of the input nodes at the entries' depths
    for (int t = 0; t < nt; ++t) {
        BatchTree& b = bp.trees[t];
        item_off[t] = (int)items.size();
        for (int i = b.obegin; i < b.oend; ++i) items.push_back(Item{t, i});
        Tree& o = *b.out;
        Tree& in = *b.inp;
        BTree& d = bt[t];
        d.okey = o.key;
        d.ocoef = o.coef;
        d.onorm2 = o.norm2;
        d.ownorm2 = o.wnorm2;
        d.in = InView{in.hkey, in.hval, in.hcap, in.coef, in.norm2};
        d.inkey = in.key;
        d.deltas = b.tab->d_deltas;
        d.terms = b.tab->d_terms;
        d.mats = b.tab->d_mats;
        d.mats32 = b.tab->d_mats32;
        d.matsD = b.tab->d_matsD;
        d.matsE = b.tab->d_matsE;
        d.matsT32 = b.tab->d_matsT32;
        d.matsbT32 = b.tab->d_matsbT32;
        d.matsI = b.tab->d_matsI;
        d.matsbI = b.tab->d_matsbI;
        d.matsS32 = b.tab->d_matsS32;
        d.matsbS32 = b.tab->d_matsbS32;
        d.matsX = b.tab->d_matsX;
        d.nprefix = b.nprefix;
        d.root = b.depth == 0;
        d.theta = b.theta;
        // split threshold: deeper entries from the root pass's norm; root entries get theirs on the device
        d.thr = b.depth == 0 ? 0.0
                             : ((b.prec > 0.0 && b.g0 > 0.0) ? b.prec * b.g0 * std::pow(2.0, -0.5 * b.depth) : INFINITY);
        d.depth = b.depth;
        d.depth_limit = m.depth_limit;
        for (int q = 0; q < 3; ++q) d.ext[q] = (long long)m.boxes[q] << b.depth;
        d.img_lb = d.img_le = 0;
        if (in.levels() > b.depth) {
            d.img_lb = in.level_begin[b.depth];
            d.img_le = in.level_begin[b.depth + 1];
        }
        d.img_base = nreal;
        nreal += d.img_le - d.img_lb;
    }
    item_off[nt] = (int)items.size();
    const int ni = (int)items.size();
    bp.nitems = ni;
    if (ni == 0) return;
    // everything the pass takes from the host, in one transfer
    std::vector<double> precs(nt);
    std::vector<ImgSrc> srcs(nt);
    bool any_root = false;
    for (int t = 0; t < nt; ++t) {
        precs[t] = bp.trees[t].prec;
        srcs[t] = ImgSrc{bp.trees[t].inp->coef, bt[t].img_base, bt[t].img_lb, bt[t].img_le - bt[t].img_lb};
        any_root |= bp.trees[t].depth == 0;
    }
    UploadPack up(ctx);
    const size_t o_items = up.add(items), o_trees = up.add(bt), o_off = up.add(item_off), o_prec = up.add(precs), o_src = up.add(srcs);
    char* d_up = up.send();
    Item* d_items = reinterpret_cast<Item*>(d_up + o_items);
    BTree* d_trees = reinterpret_cast<BTree*>(d_up + o_trees);
    int* d_item_off = reinterpret_cast<int*>(d_up + o_off);
    const double* d_prec = reinterpret_cast<const double*>(d_up + o_prec);
    const ImgSrc* d_srcs = reinterpret_cast<const ImgSrc*>(d_up + o_src);
    // the pass's counters and flags, cleared together
    struct Counters {
        unsigned long long ntrip;  // contracted triples
        int kerr, pad;             // set by the contraction on a wait timeout
        int ngreq, ngreq2, terr;   // generated-node requests (counted, numbered), the expansion's error word
    };
    Counters* d_cnt = (Counters*)dalloc(ctx, sizeof(Counters));
    MWB_CUDA(cudaMemsetAsync(d_cnt, 0, sizeof(Counters), s));
    unsigned long long* d_ntrip_tot = &d_cnt->ntrip;
    int *d_kerr = &d_cnt->kerr, *d_ngreq = &d_cnt->ngreq, *d_terr = &d_cnt->terr;

    // 1. candidates; per item: candidate and chunk counts with their sums, split flags
    unsigned long long* d_nchunk = (unsigned long long*)dalloc(ctx, (sizeof(unsigned long long) * 2 + sizeof(int) * 3) * (ni + 1));
    unsigned long long* d_choff = d_nchunk + (ni + 1);
    int* d_count = reinterpret_cast<int*>(d_choff + (ni + 1));
    int* d_offs = d_count + (ni + 1);
    int* d_sflags = d_offs + (ni + 1);
    k_bcand<<<ni, kCandThreads, 0, s>>>(d_items, d_trees, d_count, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, d_ngreq);
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    scan_only(ctx, d_count, d_offs, ni);
    int tot0[2] = {0, 0};  // candidates, generated-node requests: one read-back
    readback(ctx, {{&tot0[0], d_offs + ni, sizeof(int)}, {&tot0[1], d_ngreq, sizeof(int)}});
    const int ncand = tot0[0];
    const int ngreq = tot0[1];
    const int ncap = std::max(1, ncand);
    uint64_t* d_greq_key = (uint64_t*)dalloc(ctx, (sizeof(uint64_t) + 6 * sizeof(int)) * (ncap + 1));
    int* d_greq_leaf = reinterpret_cast<int*>(d_greq_key + (ncap + 1));
    int* d_cdelta = d_greq_leaf + (ncap + 1);
    int* d_csrc = d_cdelta + (ncap + 1);
    int* d_cand_item = d_csrc + (ncap + 1);
    int* d_ntrip = d_cand_item + (ncap + 1);
    int* d_toff = d_ntrip + (ncap + 1);
    if (ncand > 0) {
        k_bcand<<<ni, kCandThreads, 0, s>>>(d_items, d_trees, d_count, d_offs, d_cdelta, d_csrc, d_cand_item, d_greq_key,
                                            d_greq_leaf, &d_cnt->ngreq2);
        MWB_CUDA(cudaGetLastError());
        count(ctx);
    }

    // 2. generated nodes
    int nu = 0;
    uint64_t* d_ukey = nullptr;
    int* d_uleaf = nullptr;
    double* d_gblk = nullptr;
    double* d_gnorm2 = nullptr;
    if (ngreq > 0) {
        uint64_t* d_sk = (uint64_t*)dalloc(ctx, sizeof(uint64_t) * ngreq);
        int* d_sl = (int*)dalloc(ctx, sizeof(int) * ngreq);
        size_t tmp = 0;
        MWB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, d_greq_key, d_sk, d_greq_leaf, d_sl, ngreq, 0, 64, s));
        void* d_tmp = dalloc(ctx, tmp);
        MWB_CUDA(cub::DeviceRadixSort::SortPairs(d_tmp, tmp, d_greq_key, d_sk, d_greq_leaf, d_sl, ngreq, 0, 64, s));
        dfree(ctx, d_tmp);
        int* d_flags = (int*)dalloc(ctx, sizeof(int) * (ngreq + 1));
        int* d_pos = (int*)dalloc(ctx, sizeof(int) * (ngreq + 1));
        k_bunique_flags<<<(ngreq + 255) / 256, 256, 0, s>>>(d_sk, ngreq, d_flags);
        nu = scan_total(ctx, d_flags, d_pos, ngreq);
        d_ukey = (uint64_t*)dalloc(ctx, sizeof(uint64_t) * nu);
        d_uleaf = (int*)dalloc(ctx, sizeof(int) * nu);
        k_bunique_scatter<<<(ngreq + 255) / 256, 256, 0, s>>>(d_sk, d_sl, d_flags, d_pos, ngreq, d_ukey, d_uleaf);
        k_bresolve_gen<<<(ncand + 255) / 256, 256, 0, s>>>(d_csrc, ncand, d_greq_key, d_ukey, nu);
        MWB_CUDA(cudaGetLastError());
        d_gblk = (double*)dalloc(ctx, sizeof(double) * (size_t)nu * K * K * K);
        d_gnorm2 = (double*)dalloc(ctx, sizeof(double) * nu);
#define L_GEN(KK)                                                                                                        \
    {                                                                                                                    \
        MWB_CUDA(cudaFuncSetAttribute(k_bgenerate<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GenCfg<KK>::SMEM)); \
        k_bgenerate<KK><<<nu, BX<KK, KK>::NTHR, GenCfg<KK>::SMEM, s>>>(d_ukey, d_uleaf, d_trees, m.d_frH, d_gblk, d_gnorm2); \
    }
        MWB_DISPATCH_K(K, L_GEN)
#undef L_GEN
        MWB_CUDA(cudaGetLastError());
        count(ctx, 4);
        dfree(ctx, d_sk);
        dfree(ctx, d_sl);
        dfree(ctx, d_flags);
        dfree(ctx, d_pos);
    }

    // 3-4. triples per candidate, chunks
    const bool pencil = contraction_pencil();
    // the split-TF32 engine's error floor (about 2e-7 relative, data in two TF32 pieces) stays below the
    // requested precision only from prec = 1e-6 up: finer requests take the FP32 engine
    bool tc_prec_ok = true;
    for (const BatchTree& b : bp.trees) tc_prec_ok &= !(b.prec > 0.0 && b.prec < kTensorCoreMinPrec);
    // the GEMM-tiled engine runs the line-ordered contraction (chunks of sorted triples); the
    // tensor-core and pencil engines take chunks of whole candidates
    bool lined = false, lined32 = false, hyb = false;
    const bool fp64 = !pencil && bp.precision == 0;
#define L_ENG(KK)                                                                                    \
    hyb = !pencil && bp.precision == 3 && HCfg<KK>::FITS;                                            \
    lined32 = !pencil && !hyb && bp.precision >= 1 && GCfg<KK>::FITS &&                              \
              !(bp.precision == 2 && TCfg<KK>::FITS && tc_prec_ok);                                  \
    lined = fp64 || hyb || lined32;
    MWB_DISPATCH_K(K, L_ENG)
#undef L_ENG
    if (ncand > 0) {
        k_bterms<<<(ncand + 255) / 256, 256, 0, s>>>(d_cand_item, ncand, d_items, d_trees, d_cdelta, d_csrc, d_gnorm2,
                                                     d_ntrip);
        MWB_CUDA(cudaGetLastError());
        count(ctx);
    }
    const int chunk_limit = ctx->chunk_triples[std::min(std::max(bp.precision, 0), 3)];
    unsigned long long *d_tri = nullptr, *d_tkey = nullptr, *d_tval = nullptr;
    void* d_ximg = nullptr;
    int nchunks = 0, nslots = 0;
    Chunk* d_chunks = nullptr;
    if (lined) {
        const int ntri = scan_total(ctx, d_ntrip, d_toff, ncand);
        const size_t tcap = (size_t)std::max(1, ntri);
        // the sorted triples stay for the contraction, the unsorted ones go before its partial blocks are allocated
        d_tri = (unsigned long long*)dalloc(ctx, 2 * sizeof(unsigned long long) * tcap);
        unsigned long long* d_tkey_in = (unsigned long long*)dalloc(ctx, 2 * sizeof(unsigned long long) * tcap);
        unsigned long long* d_tval_in = d_tkey_in + tcap;
        d_tkey = d_tri;
        d_tval = d_tri + tcap;
        if (ntri > 0) {
            k_texpand<<<(ncand + 255) / 256, 256, 0, s>>>(d_offs, d_cand_item, ncand, d_items, d_trees, d_cdelta, d_ntrip,
                                                          d_toff, d_csrc, d_tkey_in, d_tval_in, d_terr);
            MWB_CUDA(cudaGetLastError());
            int hb = 1;
            while (hb < 31 && (1ll << hb) < (long long)ni) ++hb;
            size_t tmp = 0;
            MWB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, d_tkey_in, d_tkey, d_tval_in, d_tval, ntri, 0, 32 + hb, s));
            void* d_tmp = dalloc(ctx, tmp);
            MWB_CUDA(cub::DeviceRadixSort::SortPairs(d_tmp, tmp, d_tkey_in, d_tkey, d_tval_in, d_tval, ntri, 0, 32 + hb, s));
            dfree(ctx, d_tmp);
            count(ctx, 2);
        }
        dfree(ctx, d_tkey_in);
        k_tchunks<<<(ni * 32 + 127) / 128, 128, 0, s>>>(d_offs, d_toff, ni, d_tkey, chunk_limit, 0, d_nchunk, nullptr, nullptr);
        count(ctx);
        scan_only(ctx, d_nchunk, d_choff, ni);
        unsigned long long tot = 0;  // chunks, partial slots
        int terr = 0;                // the expansion's error word: one read-back
        readback(ctx, {{&tot, d_choff + ni, sizeof(tot)}, {&terr, d_terr, sizeof(int)}});
        if (terr != 0) throw Error(-3, "input tree nodes are not in level order");
        nchunks = (int)(uint32_t)tot;
        nslots = (int)(tot >> 32);
        d_chunks = (Chunk*)dalloc(ctx, sizeof(Chunk) * std::max(1, nchunks));
        k_tchunks<<<(ni * 32 + 127) / 128, 128, 0, s>>>(d_offs, d_toff, ni, d_tkey, chunk_limit, 1, d_nchunk, d_choff, d_chunks);
        // block images of this pass's input nodes (the entries' depth levels) and generated nodes
        const long long nimg = nreal + nu;
        if (nimg > 0) {
#define L_IMG(KK)                                                                                               \
    {                                                                                                           \
        if (hyb) {                                                                                              \
            d_ximg = launch_simage<KK>(ctx, nimg, d_srcs, nt, d_gblk, nreal, s);                                \
        } else if (lined32) {                                                                                   \
            d_ximg = dalloc(ctx, sizeof(float) * (size_t)nimg * GCfg<KK>::IMG);                                 \
            const int smem = (int)(sizeof(float) * 8 * KK * KK * KK);                                          \
            MWB_CUDA(cudaFuncSetAttribute(k_ximage<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));    \
            k_ximage<KK><<<(unsigned)nimg, 256, smem, s>>>(d_srcs, nt, d_gblk, nreal, (float*)d_ximg);           \
        } else {                                                                                                \
            d_ximg = dalloc(ctx, sizeof(double) * (size_t)nimg * DCfg<KK>::IMG);                                \
            k_dimage<KK><<<(unsigned)nimg, 256, 0, s>>>(d_srcs, nt, d_gblk, nreal, (double*)d_ximg);             \
        }                                                                                                       \
    }
            MWB_DISPATCH_K(K, L_IMG)
#undef L_IMG
            MWB_CUDA(cudaGetLastError());
            count(ctx);
        }
    } else {
        k_bchunks<<<(ni + 127) / 128, 128, 0, s>>>(d_offs, ni, d_ntrip, chunk_limit, 0, d_nchunk, nullptr, nullptr);
        count(ctx);
        scan_only(ctx, d_nchunk, d_choff, ni);
        unsigned long long tot = 0;
        readback(ctx, {{&tot, d_choff + ni, sizeof(tot)}});
        nchunks = (int)(uint32_t)tot;
        nslots = (int)(tot >> 32);
        d_chunks = (Chunk*)dalloc(ctx, sizeof(Chunk) * std::max(1, nchunks));
        k_bchunks<<<(ni + 127) / 128, 128, 0, s>>>(d_offs, ni, d_ntrip, chunk_limit, 1, d_nchunk, d_choff, d_chunks);
    }
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    double* d_partials = (double*)dalloc(ctx, sizeof(double) * BS * std::max(1, nslots));
    // the line-ordered engines (tensor-core and CUDA-core) run a copy of the chunk list sorted longest
    // first, so that a launch's last wave of CTAs holds the short chunks (the reduction keeps reading the
    // list in item order)
    Chunk* d_run = d_chunks;
    if (lined && nchunks > 1) {
        int* d_len = (int*)dalloc(ctx, sizeof(int) * 2 * (size_t)nchunks);
        d_run = (Chunk*)dalloc(ctx, sizeof(Chunk) * (size_t)nchunks);
        k_chunk_len<<<(nchunks + 255) / 256, 256, 0, s>>>(d_chunks, nchunks, d_len);
        size_t tmp = 0;
        MWB_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, d_len, d_len + nchunks, d_chunks, d_run, nchunks,
                                                           0, 16, s));
        void* d_tmp = dalloc(ctx, tmp);
        MWB_CUDA(cub::DeviceRadixSort::SortPairsDescending(d_tmp, tmp, d_len, d_len + nchunks, d_chunks, d_run, nchunks,
                                                           0, 16, s));
        dfree(ctx, d_tmp);
        dfree(ctx, d_len);
        count(ctx, 2);
    }

    // 5. contraction + reduction of multi-chunk nodes
    if (ctx->prof) MWB_CUDA(cudaEventRecord(ctx->ev0, s));
#define L_AP(KK)                                                                                             \
    {                                                                                                        \
        if (hyb) {                                                                                           \
            launch_happly<KK>(nchunks, d_run, d_items, d_trees, d_tkey, d_tval, d_csrc,                      \
                              (const unsigned char*)d_ximg, nreal, d_partials, d_ntrip_tot, d_kerr, s);       \
        } else if (bp.precision == 2 && TCfg<KK>::FITS && !pencil && tc_prec_ok) {                           \
            size_t smem = TCfg<KK>::SMEM;                                                                    \
            MWB_CUDA(cudaFuncSetAttribute(k_tapply<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
            k_tapply<KK><<<nchunks, TCfg<KK>::NTHR, smem, s>>>(d_chunks, d_items, d_trees, d_cdelta, d_csrc,     \
                                                               d_gblk, d_gnorm2, d_partials, d_ntrip_tot, d_kerr); \
        } else if (fp64) {                                                                                   \
            size_t smem = DCfg<KK>::SMEM;                                                                    \
            MWB_CUDA(cudaFuncSetAttribute(k_dapply<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
            k_dapply<KK><<<nchunks, DCfg<KK>::NTHR, smem, s>>>(d_run, d_items, d_trees, d_tkey, d_tval, d_csrc,  \
                                                               (const double*)d_ximg, nreal, d_partials,         \
                                                               d_ntrip_tot);                                     \
        } else if (lined32) {                                                                                \
            size_t smem = GCfg<KK>::SMEM;                                                                    \
            MWB_CUDA(cudaFuncSetAttribute(k_gapply<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
            k_gapply<KK><<<nchunks, GCfg<KK>::NTHR, smem, s>>>(d_run, d_items, d_trees, d_tkey, d_tval, d_csrc,  \
                                                               (const float*)d_ximg, nreal, d_partials,          \
                                                               d_ntrip_tot);                                     \
        } else if (bp.precision >= 1) {                                                                      \
            size_t smem = ACfg<KK, float>::SMEM;                                                             \
            MWB_CUDA(cudaFuncSetAttribute(k_bapply<KK, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
            k_bapply<KK, float><<<nchunks, ACfg<KK, float>::NT, smem, s>>>(d_chunks, d_items, d_trees, d_cdelta,  \
                                                                            d_csrc, d_gblk, d_gnorm2, d_partials, \
                                                                            d_ntrip_tot);                         \
        } else {                                                                                             \
            size_t smem = ACfg<KK, double>::SMEM;                                                            \
            MWB_CUDA(cudaFuncSetAttribute(k_bapply<KK, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
            k_bapply<KK, double><<<nchunks, ACfg<KK, double>::NT, smem, s>>>(d_chunks, d_items, d_trees, d_cdelta, \
                                                                              d_csrc, d_gblk, d_gnorm2, d_partials, \
                                                                              d_ntrip_tot);                        \
        }                                                                                                    \
    }
    MWB_DISPATCH_K(K, L_AP)
#undef L_AP
    MWB_CUDA(cudaGetLastError());
    if (ctx->prof) MWB_CUDA(cudaEventRecord(ctx->ev1, s));
    if (d_run != d_chunks) dfree(ctx, d_run);
    count(ctx);
    ctx->apply_launches++;
    ctx->apply_ctas += nchunks;
    if (nslots > 0) {  // one block per item; items whose node took one chunk leave at once
#define L_RED(KK) k_breduce<KK><<<ni, 256, 0, s>>>(d_chunks, d_choff, d_items, d_trees, d_partials);
        MWB_DISPATCH_K(K, L_RED)
#undef L_RED
        MWB_CUDA(cudaGetLastError());
        count(ctx);
    }

    // 6. root norms and thresholds (root entries), split flags; one read-back for the pass's results
    double* d_g = nullptr;
    if (any_root) {
        d_g = (double*)dalloc(ctx, sizeof(double) * nt);
        k_root_thr<<<nt, 256, 0, s>>>(d_items, d_item_off, d_trees, d_prec, d_g);
        MWB_CUDA(cudaGetLastError());
        count(ctx);
    }
    k_bsplit_flags<<<(ni + 255) / 256, 256, 0, s>>>(d_items, ni, d_trees, d_sflags);
    MWB_CUDA(cudaGetLastError());
    count(ctx);
    unsigned long long ntot[2] = {0, 0};
    std::vector<int> sflags(ni);
    std::vector<double> g(any_root ? nt : 0);
    readback(ctx, {{ntot, d_ntrip_tot, sizeof(ntot)}, {sflags.data(), d_sflags, sizeof(int) * ni},
                   {g.data(), d_g, any_root ? sizeof(double) * nt : 0}});
    if ((ntot[1] & 0xffffffffull) != 0)
        throw Error(-2, "contraction: an MMA or copy completion wait exceeded its time limit");
    if (ctx->prof) {
        float ms = 0.0f;
        MWB_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
        ctx->apply_ms += ms;
    }
    bp.triples = (long long)ntot[0];
    for (int t = 0; t < nt; ++t)
        if (bp.trees[t].depth == 0) bp.trees[t].g0 = std::sqrt(g[t]);
    bp.split_lists.assign(nt, {});
    for (int t = 0; t < nt; ++t)
        for (int i = item_off[t]; i < item_off[t + 1]; ++i)
            if (sflags[i]) bp.split_lists[t].push_back(items[i].node);
    dfree(ctx, d_g);
    for (void* p : std::initializer_list<void*>{d_up, d_cnt, d_nchunk, d_greq_key, d_ukey, d_uleaf, d_gblk, d_gnorm2, d_chunks,
                                                d_partials, d_tri, d_ximg})
        dfree(ctx, p);
    bp.nchunks = nchunks;
    bp.nslots = nslots;
}

}  // namespace mwb
