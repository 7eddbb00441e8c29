// mw_block.cuh -- separable transform of one (2k)^3 FP64 node block on the FP64 matrix instruction, in place in
// shared memory:  out = (Mz (x) My (x) Mx) in  with RO x 2k matrices (RO = 2k: projection, compression,
// reconstruction, point values; RO = k: one level of the descent to a node generated below its ancestor).  The input's
// wavelet half may be absent (NI = k).
//
// Bound by the FP64 pipe.  The pencil form (a thread per pencil, one operator element read from shared memory per
// FMA) ran at the shared-memory rate, a quarter of it.  Here a warp takes whole z slices: the x product's C
// fragment is the A operand of the y product (its two values per lane are the columns 2i and 2i + 1 of a
// tile: two A fragments of four b each), so x and y need no exchange and overwrite the slice where it lies; after one
// barrier the z product takes column tiles, whose columns only their own warp reads and writes.
//
// Shared layout: element (a, b, c) at a + LDA b + LDP c.  LDP (and LDA, where that costs nothing) keep the
// fragments' four-row accesses on distinct banks.  Operators are read as fragments, lane 4 n + i:
//   A order [step s][row tile r]:  M[8 r + n][4 s + i]
//   B order [column tile j][step s = 2 t + e]:  M[8 j + 4 (n mod 2) + n / 2][b], b = 8 t + 2 i + e, or 8 t + i in a
//   last tile of at most four (one step then covers it)
// zero outside the matrix.
#pragma once
#include "mw_device.cuh"

namespace mwb {

template <int K, int RO>
struct BX {
    static constexpr int K2 = 2 * K;
    static constexpr int S = (K2 + 3) / 4, CT = (K2 + 7) / 8, FT = K2 / 8, REM = K2 % 8;
    static constexpr bool HALF = REM != 0 && REM <= 4;  // a last tile of at most four columns
    static constexpr int RT = (RO + 7) / 8;
    static constexpr int LDA = K2 == 16 ? 20 : K2;  // input rows
    static constexpr int LDO = RO == 16 ? 20 : RO;  // output rows
    static constexpr int NZT = (RO * RO + 7) / 8;
    __host__ __device__ static constexpr int physo(int n) { return LDO == RO ? n : n + (LDO - RO) * (n / RO); }
    static constexpr int LDP = dcfg_ld(LDA == K2 ? (K2 * K2 + 7) / 8 * 8 : LDA * K2);
    static constexpr int VOL = LDP * K2;
    static constexpr int FRAG = S * RT * 32;  // one operator
    // A warp belongs to one SM sub-partition: with k warps of two slices each, k = 9, 10 loads two of the four half as much
    // again as the others, eight warps with slices dealt in turn load them evenly (28 pair products: k = 9 8.80 -> 8.07 ms,
    // k = 10 8.08 -> 7.82, k = 11 10.95 -> 10.77; k = 5, 6, 7 do not gain).  The sums' kernel (RO = k) holds a block in
    // registers and needs the threads (k = 11: 4 % slower with eight warps).
    static constexpr int NWARP = RO == K2 && K >= 9 && K <= 11 ? 8 : K, NTHR = 32 * NWARP;
};

// b of column n of an x tile (>= 2k: padding)
template <int K, int RO>
__host__ __device__ constexpr int bx_col(int t, int n) {
    using C = BX<K, RO>;
    return C::HALF && t == C::FT ? 8 * t + (n >> 1) : 8 * t + n;
}
// fragments of a row-major RO x 2k matrix (entry(o, i)); e = position within the operator's FRAG doubles
template <int K, int RO, typename F>
__host__ __device__ inline double bx_frag_a(int e, F&& entry) {
    using C = BX<K, RO>;
    const int lane = e & 31, q = e >> 5, o = 8 * (q % C::RT) + (lane >> 2), i = 4 * (q / C::RT) + (lane & 3);
    return o < RO && i < C::K2 ? entry(o, i) : 0.0;
}
template <int K, int RO, typename F>
__host__ __device__ inline double bx_frag_b(int e, F&& entry) {
    using C = BX<K, RO>;
    const int lane = e & 31, q = e >> 5, n = lane >> 2, i = lane & 3, s = q % C::S, t = s / 2;
    const int o = 8 * (q / C::S) + 4 * (n & 1) + (n >> 1);
    const int b = C::HALF && t == C::FT ? 8 * t + i : 8 * t + 2 * i + s % 2;
    return o < RO && b < C::K2 ? entry(o, b) : 0.0;
}

// x and y products of slice c (one warp, in place): X[c][b][a] -> X[c][b'][a'], rows LDI -> LDO.  NI: the input's extent, 2k,
// or k for a scaling block alone (its wavelets zero)
template <int K, int RO, int NI = 2 * K, int LDI = BX<K, RO>::LDA>
__device__ __forceinline__ void bx_slice(double* X, int c, const double* fx, const double* fy) {
    using C = BX<K, RO>;
    constexpr int RT = C::RT, S = C::S, SI = (NI + 3) / 4, CT = (NI + 7) / 8, SY = NI == C::K2 ? S : 2 * CT;
    const int lane = threadIdx.x & 31, fi = lane & 3, fn = lane >> 2;
    double* P = X + c * C::LDP;
    double D[RT][CT][2];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int t = 0; t < CT; ++t) D[r][t][0] = D[r][t][1] = 0.0;
#pragma unroll
    for (int s = 0; s < SI; ++s) {
        double a[RT];
#pragma unroll
        for (int r = 0; r < RT; ++r) a[r] = fx[(s * RT + r) * 32 + lane];
        const int ai = 4 * s + fi;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const int b = bx_col<K, RO>(t, fn);
            const bool in = (4 * s + 3 < NI || ai < NI) && (8 * t + 7 < NI || b < NI);
            const double v = in ? P[ai + LDI * b] : 0.0;
#pragma unroll
            for (int r = 0; r < RT; ++r) dmma(D[r][t], a[r], v);
        }
    }
    __syncwarp();  // the slice is read
#pragma unroll
    for (int j = 0; j < RT; ++j) {
        double Y[RT][2];
#pragma unroll
        for (int r = 0; r < RT; ++r) Y[r][0] = Y[r][1] = 0.0;
#pragma unroll
        for (int s = 0; s < SY; ++s) {
            const double m = fy[(j * S + s) * 32 + lane];
#pragma unroll
            for (int r = 0; r < RT; ++r) dmma(Y[r], D[r][s / 2][s % 2], m);
        }
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ax = 8 * r + fn, bx = 8 * j + 4 * e + fi;
                if (ax < RO && bx < RO) P[ax + C::LDO * bx] = Y[r][e];
            }
    }
}

// z product of column tile q (one warp): v[r][h] = out at c' = 8 r + lane / 4, column 8 q + 2 (lane mod 4) + h of
// (a', b')
template <int K, int RO, int NQ, int NI = 2 * K>
__device__ __forceinline__ void bx_z(const double* X, int q0, int dq, const double* fz, double (&v)[NQ][BX<K, RO>::RT][2]) {
    using C = BX<K, RO>;
    constexpr int RT = C::RT, SI = (NI + 3) / 4;
    const int lane = threadIdx.x & 31, fi = lane & 3, fn = lane >> 2;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int r = 0; r < RT; ++r) v[q][r][0] = v[q][r][1] = 0.0;
#pragma unroll
    for (int s = 0; s < SI; ++s) {
        double a[RT];
#pragma unroll
        for (int r = 0; r < RT; ++r) a[r] = fz[(s * RT + r) * 32 + lane];
        const int c = 4 * s + fi;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int tile = q0 + q * dq;
            const double b = (4 * s + 3 < NI || c < NI) && tile < C::NZT ? X[c * C::LDP + C::physo(8 * tile) + fn] : 0.0;
#pragma unroll
            for (int r = 0; r < RT; ++r) dmma(v[q][r], a[r], b);
        }
    }
}

// every column tile of this warp, two at a time; f(c', n, v0, v1) takes the outputs (n even, and n + 1) of each lane
// (NW: the kernel's warps)
template <int K, int RO, int NI = 2 * K, int NW = BX<K, RO>::NWARP, typename F>
__device__ __forceinline__ void bx_columns(const double* X, const double* fz, F&& f) {
    using C = BX<K, RO>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = warp; q < C::NZT; q += 2 * NW) {
        double v[2][C::RT][2];
        bx_z<K, RO, 2, NI>(X, q, NW, fz, v);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int r = 0; r < C::RT; ++r) {
                const int cz = 8 * r + (lane >> 2), n = 8 * (q + h * NW) + 2 * (lane & 3);
                if (cz < RO && n < RO * RO) f(cz, n, v[h][r][0], v[h][r][1]);
            }
    }
}

// a block from global memory (x fastest) into the shared layout, asynchronously, by the NW warps of the kernel (which the kinds
// of products differ in: at k = 9 to 11 eight against k)
template <int K, int NW>
__device__ __forceinline__ void bx_load(double* X, const double* __restrict__ blk) {
    using C = BX<K, 2 * K>;
    constexpr int H = K, N = C::K2 * C::K2 * H;  // 16-byte pairs
    for (int e = threadIdx.x; e < N; e += 32 * NW) {
        const int r = e / H, i = e - r * H, b = r % C::K2, c = r / C::K2;
        cp_async16(X + 2 * i + C::LDA * b + C::LDP * c, blk + 2 * (size_t)e);
    }
    cp_async_commit();
}
// a prepared operator's fragments into shared memory
__device__ __forceinline__ void bx_operator(double* f, const double* __restrict__ img, int n, int nthr) {
    for (int e = 2 * threadIdx.x; e < n; e += 2 * nthr) cp_async16(f + e, img + e);
    cp_async_commit();
}

// Index of the deepest node on the path to `key` that a tree has, and its depth: one warp, a lane per depth
// (`key` itself included); idx < 0: none
__device__ __forceinline__ void bx_lookup(const uint64_t* hk, const int* hv, uint32_t hcap, uint64_t key, int& idx, int& depth) {
    const int lane = threadIdx.x & 31, dk = key_depth(key);
    long long t[3];
    key_trans(key, t);
    int i = -1;
    if (lane <= dk) {
        const int sh = dk - lane;
        i = hlookup(hk, hv, hcap, make_key(lane, t[0] >> sh, t[1] >> sh, t[2] >> sh));
    }
    const unsigned m = __ballot_sync(0xffffffffu, i >= 0);
    depth = m ? 31 - __clz(m) : -1;
    idx = m ? __shfl_sync(0xffffffffu, i, depth) : -1;
}

// x and y products of every slice, distributed over the kernel's NW warps; fx, fy: operators
template <int K, int RO, int NI = 2 * K, int LDI = BX<K, RO>::LDA, int NW = BX<K, RO>::NWARP>
__device__ __forceinline__ void bx_slices(double* X, const double* fx, const double* fy) {
    for (int c = threadIdx.x >> 5; c < NI; c += NW) bx_slice<K, RO, NI, LDI>(X, c, fx, fy);
}

// From an ancestor's block in X to the scaling block of the node L >= 1 levels below it along the translations t (of the
// descendant), in place with rows of k (element (a, b, c) at a + k b + LDP c): first the reconstruction's rows of the child on
// the path (k x 2k), then zero-wavelet descents (k x k).  h: their images [child bit][A, B order], in shared memory.
// Level by level: every level's rounding is relative to that level's block.  One product of the levels' matrices on the
// ancestor's block would do with fewer steps, but leaves in each descendant rounding of the size of the ancestor's largest
// values; where the function falls off inside the ancestor, a product of two such factors was noise, and refinement
// followed it down (404 nodes and growing fourfold per level against 236).
// The caller has X and h complete for every warp (a barrier), and so has it the result
template <int K, int NW>
__device__ __forceinline__ void bx_descend(double* X, const double* h, const long long (&t)[3], int L) {
    using C = BX<K, K>;
    auto img = [&](int d, int lev, int form) { return h + (2 * (int)((t[d] >> lev) & 1) + form) * C::FRAG; };
    auto put = [&](int c, int n, double v0, double v1) {
        // in the columns' own place: every lane's reads have fed the matrix instruction, which the warp executes together
        double* p = X + c * C::LDP + C::physo(n);
        p[0] = v0;
        if (n + 1 < K * K) X[c * C::LDP + C::physo(n + 1)] = v1;
    };
    bx_slices<K, K, 2 * K, C::LDA, NW>(X, img(0, L - 1, 0), img(1, L - 1, 1));
    __syncthreads();
    bx_columns<K, K, 2 * K, NW>(X, img(2, L - 1, 0), put);
    __syncthreads();
    for (int lev = L - 2; lev >= 0; --lev) {
        bx_slices<K, K, K, C::LDO, NW>(X, img(0, lev, 0), img(1, lev, 1));
        __syncthreads();
        bx_columns<K, K, K, NW>(X, img(2, lev, 0), put);
        __syncthreads();
    }
}

}  // namespace mwb
