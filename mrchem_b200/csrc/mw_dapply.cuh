// mw_dapply.cuh -- line-ordered contraction of the NS-form apply in FP64 on the FP64 matrix instruction
// (mma.sync m8n8k4; the fifth-generation tensor cores have no FP64 kind).  Included by mw_apply.cu after
// the Chunk / Item / BTree records; same contract as the other line-ordered engines: one CTA per chunk
// of one output node's triples sorted by (term, dz, dy), the sum written to the output block (or a partial
// slot) with its norms.  Every order k = 4 .. 12.
//
//   out += sum_dz beta Mz(dz) [ sum_dy My(dy) [ sum_dx Mx(dx) in_(dx,dy,dz) ] ]      (line, plane sums)
//
// What bounds it: the FP64 pipe.  The matrix instruction sustains 36.5 TFLOP/s from two warps per SM
// sub-partition (scalar FMAs 31), and takes its operands from 3 values per lane and 256 FMAs, where a
// register-tiled scalar GEMM reads 10 shared words per 25 FMAs and ran at the shared-memory rate (12.6
// TFLOP/s executed at k = 10).
//
// Work split.  Warp p owns the z-index pair (c = p, p + k): one slice of the scaling half and one of the
// wavelet half, so that generated (scaling-only) inputs and the s->s correction load every warp alike.
// The x product of its 2 x 2k columns (b, c) accumulates in registers over the line's triples (rows a',
// columns b: the FP64 C fragment), and that fragment is the A operand of the y product as it stands: a
// lane's two C values are columns 2j and 2j+1, so with columns ordered b = 8t + 4e + j (e the parity) each
// of the two values is one A fragment of four consecutive b.  Nothing is exchanged between warps, no
// barrier is needed, until a plane's y sums go to shared memory (T2) for the z product.  When 2k mod 8 is
// 2 or 4 the two slices share one column tile (even columns one slice, odd columns the other): at k = 10
// the pair's 40 columns are exactly five tiles.  Rows are padded to a multiple of 8 (2k = 20: 24).
//
// Staging.  Each warp streams its own part of the triples' block images (fragment order, one slab per
// step of four a) and of the x operators through a private ring of NS slabs by cp.async, so that no two
// warps wait for one another and the ring runs ahead across triples, lines and planes.  The y and z
// operators are read as fragments straight from global memory (L1 / L2 hits: every warp reads the same).
//
// Below the root the s->s block (T x T x T on the scaling part) is left out: the steps a < k of the
// corner tiles (a', b < k of the scaling slice) accumulate apart (S), are added to the full sums at the
// line's end, and go through their own y product into U2; the z product takes U2 off with -Tz as further
// steps of the same accumulators.  FP64 accumulators of the output block live in tensor memory between
// planes (one read and one write per plane).
#pragma once

namespace mwb {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// smallest n >= v with n mod 16 in {4, 12}: rows of doubles on four distinct groups of four banks
__host__ __device__ constexpr int dcfg_ld(int v) {
    while (v % 16 != 4 && v % 16 != 12) ++v;
    return v;
}

template <int K>
struct DCfg {
    static constexpr int K2 = 2 * K;
    static constexpr int RT = (K2 + 7) / 8;   // row tiles of an operator
    static constexpr int S = (K2 + 3) / 4;    // steps of a contraction over 2k
    static constexpr int FT = K2 / 8, REM = K2 % 8;
    static constexpr int WOFF = FT + (REM != 0 ? 1 : 0);               // first own tile of the wavelet slice
    static constexpr int NTP = 2 * FT + (REM == 0 ? 0 : REM <= 4 ? 1 : 2);  // column tiles of a pair
    static constexpr int NWARP = K, NTHR = 32 * K;
    static constexpr int RS = (K + 7) / 8;    // row and column tiles of the scaling corner
    static constexpr int KS = (K + 3) / 4;    // steps of a contraction over k
    static constexpr bool MIXED = K % 4 != 0; // the last of them also covers wavelet indices
    static constexpr int SLABX = NTP * 32, SLABA = RT * 32, SLAB = SLABX + SLABA;  // doubles
    static constexpr int MATD = S * RT * 32;           // operator image
    static constexpr int IMG = K * S * NTP * 32;       // block image
    // T2 [c][a' + PP b']: PP keeps a y fragment's stores off one another's banks where 2k does not
    // (2k = 16: four-way otherwise); at 2k = 24 shared memory has no room for it (two-way stores)
    static constexpr int PP = (K2 == 8 || K2 == 16) ? K2 + 4 : K2;
    static constexpr int NZT = (K2 * K2 + 7) / 8;      // column tiles of the z step
    __host__ __device__ static constexpr int phys(int n) { return PP == K2 ? n : n + (PP - K2) * (n / K2); }
    static constexpr int LD2 = dcfg_ld(PP == K2 ? 8 * NZT : PP * K2);
    static constexpr int LDU = dcfg_ld(PP == K2 ? (K * K2 + 7) / 8 * 8 : PP * K);
    static constexpr int ZT = (NZT + NWARP - 1) / NWARP;  // z tiles per warp (interleaved over the warps)
    static constexpr int ZD = ZT * RT * 2;                // accumulators per lane
    static constexpr int TCOLS_NEED = ((NWARP + 3) / 4) * 2 * ZD;
    static constexpr int TCOLS = TCOLS_NEED <= 32 ? 32 : TCOLS_NEED <= 64 ? 64 : TCOLS_NEED <= 128 ? 128
                                 : TCOLS_NEED <= 256 ? 256 : 512;
    // a plane's y sums in registers where they fit beside the x sums, else added up in T2
    static constexpr bool EREG = K <= 8 && K != 7;
    static constexpr int MAXT = 128;  // triples per chunk whose records are kept in shared memory
    static constexpr int MINB = K <= 4 ? 4 : K <= 5 ? 3 : K <= 8 ? 2 : 1;
    static constexpr int FIXED = 8 * (K2 * LD2 + K * LDU) + MAXT * 16;
    static constexpr int BUDGET = 232448 / MINB - 1024 - 1024;  // less the static part and the reserved part
    static constexpr int NS_FIT = (BUDGET - FIXED) / (8 * NWARP * SLAB);
    static constexpr int NS = NS_FIT > 6 ? 6 : NS_FIT;
    static constexpr size_t SMEM = FIXED + (size_t)8 * NWARP * NS * SLAB;
    static_assert(NS >= 3 && TCOLS_NEED <= 512 && MINB * TCOLS <= 512 && RS <= FT, "DCfg");
};

// (slice, b) of column n of a pair's tile j; b >= 2k: padding
template <int K>
__host__ __device__ constexpr int dcol_slice(int j, int n) {
    using C = DCfg<K>;
    if (C::REM != 0 && C::REM <= 4 && j == C::FT) return n & 1;
    return j >= C::WOFF ? 1 : 0;
}
template <int K>
__host__ __device__ constexpr int dcol_b(int j, int n) {
    using C = DCfg<K>;
    if (C::REM != 0 && C::REM <= 4 && j == C::FT) return 8 * C::FT + (n >> 1);
    const int t = j >= C::WOFF ? j - C::WOFF : j;
    return 8 * t + 4 * (n & 1) + (n >> 1);
}

// Block images of the FP64 engine, in the order the x step's B fragments are read: [pair p][step s]
// [tile couple][lane][2], then a last odd tile [lane]; lane = 4 n + i holds X[a = 4s + i][column n].  One CTA per
// block; the four lanes of a column read one 32-byte sector, writes are contiguous.  Slot numbering as
// k_ximage; a generated node's block is its k^3 scaling part.  Bound by HBM (one read, one write).
template <int K>
__global__ void __launch_bounds__(256) k_dimage(const ImgSrc* __restrict__ srcs, int nsrc, const double* __restrict__ gblk,
                                                long long nreal, double* __restrict__ img) {
    using C = DCfg<K>;
    constexpr int K2 = C::K2, NP2 = C::NTP / 2;
    const long long slot = blockIdx.x;
    const double* b;
    const bool real = slot < nreal;
    if (real) {
        int lo = 0, hi = nsrc - 1;  // last entry with base <= slot
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (srcs[mid].base <= slot) lo = mid;
            else hi = mid - 1;
        }
        const ImgSrc sr = srcs[lo];
        b = sr.coef + (size_t)(sr.lb + (slot - sr.base)) * (K2 * K2 * K2);
    } else {
        b = gblk + (size_t)(slot - nreal) * (K * K * K);
    }
    double* out = img + (size_t)slot * C::IMG;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = lane & 3, n = lane >> 2;
    auto value = [&](int p, int s, int j) -> double {
        const int a = 4 * s + i, sl = dcol_slice<K>(j, n), bb = dcol_b<K>(j, n), c = sl ? p + K : p;
        if (real) return a < K2 && bb < K2 ? b[a + K2 * (bb + K2 * c)] : 0.0;
        return a < K && bb < K && !sl ? b[a + K * (bb + K * c)] : 0.0;
    };
    for (int ps = warp; ps < K * C::S; ps += 8) {
        const int p = ps / C::S, s = ps - p * C::S;
        double* o = out + (size_t)ps * C::SLABX;
#pragma unroll
        for (int q = 0; q < NP2; ++q)
            *reinterpret_cast<double2*>(o + 64 * q + 2 * lane) = make_double2(value(p, s, 2 * q), value(p, s, 2 * q + 1));
        if constexpr (C::NTP % 2 != 0) o[64 * NP2 + lane] = value(p, s, C::NTP - 1);
    }
}

// record of one triple of a chunk (16 bytes); a matrix index fits 27 bits
struct DTri {
    int slot;  // block image slot of the input node
    int mx, my;
    unsigned mz : 27;
    unsigned flags : 5;  // DT_* below
};
static_assert(sizeof(DTri) == 16, "triple record");
enum { DT_GEN = 1, DT_LSTART = 2, DT_LEND = 4, DT_PSTART = 8, DT_PEND = 16 };

__device__ __forceinline__ void cp_async16_ca(void* smem_dst, const void* gmem_src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)),
                 "l"(gmem_src)
                 : "memory");
}

template <int K>
__global__ void __launch_bounds__(DCfg<K>::NTHR, DCfg<K>::MINB)
    k_dapply(const Chunk* __restrict__ chunks, const Item* __restrict__ items, const BTree* __restrict__ trees,
             const unsigned long long* __restrict__ tkey, const unsigned long long* __restrict__ tval,
             const int* __restrict__ csrc, const double* __restrict__ dimg, long long gbase, double* partials,
             unsigned long long* ntrip_out) {
    using C = DCfg<K>;
    constexpr int K2 = C::K2, RT = C::RT, S = C::S, NTP = C::NTP, RS = C::RS, KS = C::KS, FT = C::FT, ZT = C::ZT;
    constexpr int LD2 = C::LD2, LDU = C::LDU, PP = C::PP, NS = C::NS, SLAB = C::SLAB;
    constexpr int BS = K2 * K2 * K2;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ uint32_t tmem_slot;
    __shared__ double red[64];
    double* T2 = reinterpret_cast<double*>(smraw);  // [2k][LD2]
    double* U2 = T2 + K2 * LD2;                     // [k][LDU]
    DTri* meta = reinterpret_cast<DTri*>(U2 + K * LDU);
    double* ring0 = reinterpret_cast<double*>(meta + C::MAXT);
    const Chunk ch = chunks[blockIdx.x];
    const Item it = items[ch.item];
    const BTree& TR = trees[it.tree];
    const bool root = TR.root != 0;
    const double* __restrict__ mats = TR.matsD;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fi = lane & 3, fn = lane >> 2;  // fragment coordinates: A (row fn, k fi), B (k fi, column fn)
    const int ntri = ch.c1 - ch.c0;

    auto load_rec = [&](int t) -> DTri {
        const unsigned long long tv = tval[t];
        const int src = csrc[(int)(tv >> 32)];
        const TermRec tr = TR.terms[(int)(tv & 0xffffffffull)];
        const uint32_t lk = (uint32_t)(tkey[t] & 0xffffffffull);
        const uint32_t lp = t > ch.c0 ? (uint32_t)(tkey[t - 1] & 0xffffffffull) : ~lk;
        const uint32_t ln = t + 1 < ch.c1 ? (uint32_t)(tkey[t + 1] & 0xffffffffull) : ~lk;
        DTri h;
        h.slot = (int)(src < 0 ? gbase + (-src - 1) : TR.img_base + (src - TR.img_lb));
        h.mx = tr.mx;
        h.my = tr.my;
        h.mz = (unsigned)tr.mz;
        h.flags = (src < 0 ? DT_GEN : 0) | (lp != lk ? DT_LSTART : 0) | (ln != lk ? DT_LEND : 0) |
                  ((lp >> 10) != (lk >> 10) ? DT_PSTART : 0) | ((ln >> 10) != (lk >> 10) ? DT_PEND : 0);
        return h;
    };
    for (int e = tid; e < min(ntri, C::MAXT); e += C::NTHR) meta[e] = load_rec(ch.c0 + e);
    auto rec = [&](int t) -> DTri { return t - ch.c0 < C::MAXT ? meta[t - ch.c0] : load_rec(t); };
    for (int e = tid; e < K * LDU; e += C::NTHR) U2[e] = 0.0;  // positions outside (a', b') < k stay zero
    if (warp == 0) {
        tmem_alloc(&tmem_slot, C::TCOLS);
        tmem_relinquish();
    }
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t tacc = tmem_slot + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * 2 * C::ZD);
    {
        uint32_t z[2 * C::ZD];
#pragma unroll
        for (int q = 0; q < 2 * C::ZD; ++q) z[q] = 0u;
        tmem_span_st<0, 2 * C::ZD>(tacc, z);
        tmem_wait_st();
    }

    // ---- staging stream: slabs (triple pt, step ps) into this warp's ring, one commit group per slab
    double* ring = ring0 + (size_t)warp * NS * SLAB;
    int pt = ch.c0, ps = 0, pn = 0;
    bool pgen = false;
    const double *px = nullptr, *pa = nullptr;
    auto open = [&](int t) {
        const DTri h = rec(t);
        pgen = (h.flags & DT_GEN) != 0;
        pn = pgen ? KS : S;
        px = dimg + (size_t)h.slot * C::IMG + (size_t)warp * S * C::SLABX;
        pa = mats + (size_t)h.mx * C::MATD;
        ps = 0;
    };
    if (pt < ch.c1) open(pt);
    auto issue = [&](int slot) {
        if (pt < ch.c1) {
            double* dst = ring + slot * SLAB;
            // a generated input has columns in the first RS tiles only (the first couple of tiles holds them)
            const int nx = pgen ? 32 : C::SLABX / 2;
#pragma unroll
            for (int e = 0; e < (C::SLABX / 2 + 31) / 32; ++e)
                if (lane + 32 * e < nx) cp_async16(dst + 2 * (lane + 32 * e), px + 2 * (lane + 32 * e));
#pragma unroll
            for (int e = 0; e < (C::SLABA / 2 + 31) / 32; ++e)
                if (lane + 32 * e < C::SLABA / 2)
                    cp_async16_ca(dst + C::SLABX + 2 * (lane + 32 * e), pa + 2 * (lane + 32 * e));
            px += C::SLABX;
            pa += C::SLABA;
            if (++ps == pn && ++pt < ch.c1) open(pt);
        }
        cp_async_commit();
    };
    int slot = 0;
#pragma unroll 1
    for (int q = 0; q < NS - 1; ++q) issue(q);

    double D[RT][NTP][2];                       // x sums of the line (the corner's steps a >= k)
    double SC[RS][RS][2];                       // ... and the corner's steps a < k
    double E[C::EREG ? 2 : 1][RT][RT][2];       // y sums: rows a', columns b' = 8 t + 4 e + fi
    bool line_gen = true, plane_gen = true, first_line = true;
    for (int t = ch.c0; t < ch.c1; ++t) {
        const DTri h = rec(t);
        const bool gen = (h.flags & DT_GEN) != 0;
        if (h.flags & DT_PSTART) {
            plane_gen = true;
            first_line = true;
        }
        if (h.flags & DT_LSTART) {
            line_gen = true;
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int j = 0; j < NTP; ++j) D[r][j][0] = D[r][j][1] = 0.0;
#pragma unroll
            for (int r = 0; r < RS; ++r)
#pragma unroll
                for (int j = 0; j < RS; ++j) SC[r][j][0] = SC[r][j][1] = 0.0;
        }
        line_gen = line_gen && gen;
        plane_gen = plane_gen && gen;
        // ---- x: D[a'][(b, c)] += sum_a Mx[a'][a] X[a][(b, c)]
#pragma unroll
        for (int s = 0; s < S; ++s) {
            if (s >= KS && gen) break;
            cp_async_wait_group<NS - 2>();
            __syncwarp();  // the slab is in for every lane, and every lane has read the previous one
            issue(slot == 0 ? NS - 1 : slot - 1);
            const double* sx = ring + slot * SLAB;
            slot = slot + 1 == NS ? 0 : slot + 1;
            double a[RT];
#pragma unroll
            for (int r = 0; r < RT; ++r) a[r] = sx[C::SLABX + 32 * r + lane];
            double b[NTP + 1];
            {
                const double2 v = *reinterpret_cast<const double2*>(sx + 2 * lane);
                b[0] = v.x;
                b[1] = v.y;
            }
            const bool mixed = C::MIXED && s == KS - 1;
#pragma unroll
            for (int j = 0; j < RS; ++j)
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    if (r < RS && s < KS) {
                        if (mixed) {
                            const bool sa = 4 * s + fi < K;
                            dmma(SC[r][j], sa ? a[r] : 0.0, b[j]);
                            if (!gen) dmma(D[r][j], sa ? 0.0 : a[r], b[j]);
                        } else {
                            dmma(SC[r][j], a[r], b[j]);
                        }
                    } else {
                        dmma(D[r][j], a[r], b[j]);
                    }
                }
            if (!gen) {
#pragma unroll
                for (int q = 1; q < NTP / 2; ++q) {
                    const double2 v = *reinterpret_cast<const double2*>(sx + 64 * q + 2 * lane);
                    b[2 * q] = v.x;
                    b[2 * q + 1] = v.y;
                }
                if constexpr (NTP % 2 != 0) b[NTP - 1] = sx[64 * (NTP / 2) + lane];
#pragma unroll
                for (int j = RS; j < NTP; ++j)
#pragma unroll
                    for (int r = 0; r < RT; ++r) dmma(D[r][j], a[r], b[j]);
            }
        }
        if (!(h.flags & DT_LEND)) continue;
        if (first_line) __syncthreads();  // the previous plane's z step has read T2 and U2
#pragma unroll
        for (int r = 0; r < RS; ++r)
#pragma unroll
            for (int j = 0; j < RS; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) D[r][j][e] += SC[r][j][e];
        // ---- y: E[a'][b'] (+)= sum_b D[a'][b] beta My[b'][b]   (a plane sums its lines)
        const double beta = TR.matsDbeta[h.my];
        // lane's element of the operator image as a B fragment: row b' = 8 t + 4 (fn & 1) + (fn >> 1)
        const double* my = mats + (size_t)h.my * C::MATD + 4 * (4 * (fn & 1) + (fn >> 1)) + fi;
#pragma unroll
        for (int sl = 0; sl < 2; ++sl) {
            constexpr bool ER = C::EREG;
            auto& Es = E[ER ? sl : 0];
            const int c = sl ? warp + K : warp;
            double* t2 = T2 + c * LD2 + fn + PP * fi;
            auto t2at = [&](int r, int j, int e) -> double* { return t2 + 8 * r + PP * (8 * j + 4 * e); };
            auto inside = [&](int r, int j, int e) { return 8 * r + fn < K2 && 8 * j + 4 * e + fi < K2; };
            if (ER ? first_line : true) {
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int j = 0; j < RT; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            Es[r][j][e] = (ER || first_line || !inside(r, j, e)) ? 0.0 : *t2at(r, j, e);
            }
            if (!(sl == 1 && line_gen)) {
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    if (s >= KS && line_gen) break;
                    double m[RT];
#pragma unroll
                    for (int j = 0; j < RT; ++j) m[j] = beta * __ldg(my + (s * RT + j) * 32);
                    // step s = 2 t + e of the slice: parity e of its tile t, or its parity of the shared tile
                    constexpr bool SH = C::REM != 0 && C::REM <= 4;
                    const int tile = (SH && s == 2 * FT) ? FT : (sl ? C::WOFF : 0) + s / 2;
                    const int e = (SH && s == 2 * FT) ? sl : s % 2;
#pragma unroll
                    for (int r = 0; r < RT; ++r)
#pragma unroll
                        for (int j = 0; j < RT; ++j) dmma(Es[r][j], D[r][tile][e], m[j]);
                }
            }
            if (ER ? (h.flags & DT_PEND) != 0 : true) {
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int j = 0; j < RT; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (inside(r, j, e)) *t2at(r, j, e) = Es[r][j][e];
            }
        }
        if (!root) {  // s->s: U2[a'][b'] (+)= sum_{b<k} SC[a'][b] beta Ty[b'][b]
            double ES[RS][RS][2];
            double* u = U2 + warp * LDU + fn + PP * fi;
            auto inside = [&](int r, int j, int e) { return 8 * r + fn < K && 8 * j + 4 * e + fi < K; };
#pragma unroll
            for (int r = 0; r < RS; ++r)
#pragma unroll
                for (int j = 0; j < RS; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        ES[r][j][e] = (!first_line && inside(r, j, e)) ? u[8 * r + PP * (8 * j + 4 * e)] : 0.0;
#pragma unroll
            for (int s = 0; s < KS; ++s)
#pragma unroll
                for (int j = 0; j < RS; ++j) {
                    const double m = 4 * s + fi < K ? beta * __ldg(my + (s * RT + j) * 32) : 0.0;
#pragma unroll
                    for (int r = 0; r < RS; ++r) dmma(ES[r][j], SC[r][s / 2][s % 2], m);
                }
#pragma unroll
            for (int r = 0; r < RS; ++r)
#pragma unroll
                for (int j = 0; j < RS; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (inside(r, j, e)) u[8 * r + PP * (8 * j + 4 * e)] = ES[r][j][e];
        }
        first_line = false;
        if (!(h.flags & DT_PEND)) continue;
        __syncthreads();  // the plane's y sums are in T2, U2
        // ---- z: acc[c'][(a', b')] += sum_c Mz[c'][c] T2[c][(a', b')]  - the s->s block
        {
            uint32_t w[2 * C::ZD];
            tmem_span_ld<0, 2 * C::ZD>(tacc, w);
            tmem_span_wait<0, 2 * C::ZD>(w);
            double z[ZT][RT][2];
#pragma unroll
            for (int q = 0; q < C::ZD; ++q) z[q / (2 * RT)][(q / 2) % RT][q % 2] = words_to_double(w[2 * q], w[2 * q + 1]);
            const double* mz = mats + (size_t)h.mz * C::MATD + lane;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (s >= KS && plane_gen) break;
                double a[RT];
#pragma unroll
                for (int r = 0; r < RT; ++r) a[r] = __ldg(mz + (s * RT + r) * 32);
                const int c = 4 * s + fi;
#pragma unroll
                for (int q = 0; q < ZT; ++q) {
                    const int tile = warp + C::NWARP * q;
                    if (tile < C::NZT) {
                        const double b = (4 * s + 3 < K2 || c < K2) ? T2[c * LD2 + C::phys(8 * tile) + fn] : 0.0;
#pragma unroll
                        for (int r = 0; r < RT; ++r) dmma(z[q][r], a[r], b);
                    }
                }
                if (s < KS && !root) {
                    double ac[RS];
#pragma unroll
                    for (int r = 0; r < RS; ++r) ac[r] = (8 * r + fn < K && c < K) ? -a[r] : 0.0;
#pragma unroll
                    for (int q = 0; q < ZT; ++q) {
                        const int n0 = 8 * (warp + C::NWARP * q);  // columns with some a', b' < k
                        if (n0 < K * K2 && (n0 % K2 < K || n0 % K2 + 7 >= K2)) {
                            const double b = (4 * s + 3 < K || c < K) ? U2[c * LDU + C::phys(n0) + fn] : 0.0;
#pragma unroll
                            for (int r = 0; r < RS; ++r) dmma(z[q][r], ac[r], b);
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < C::ZD; ++q)
                double_to_words(z[q / (2 * RT)][(q / 2) % RT][q % 2], w[2 * q], w[2 * q + 1]);
            tmem_span_st<0, 2 * C::ZD>(tacc, w);
            tmem_wait_st();
        }
    }
    cp_async_wait_all();
    double* dst = ch.slot < 0 ? TR.ocoef + (size_t)it.node * BS : partials + (size_t)ch.slot * BS;
    double n2 = 0.0, w2 = 0.0;
    {
        uint32_t w[2 * C::ZD];
        tmem_span_ld<0, 2 * C::ZD>(tacc, w);
        tmem_span_wait<0, 2 * C::ZD>(w);
#pragma unroll
        for (int q = 0; q < ZT; ++q)
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                const int cz = 8 * r + fn, n = 8 * (warp + C::NWARP * q) + 2 * fi;
                if (cz < K2 && n < K2 * K2) {  // 2k is even: n and n + 1 lie in one row of the block
                    const int i = 2 * ((q * RT + r) * 2);
                    const double v0 = words_to_double(w[i], w[i + 1]), v1 = words_to_double(w[i + 2], w[i + 3]);
                    *reinterpret_cast<double2*>(dst + (size_t)cz * K2 * K2 + n) = make_double2(v0, v1);
                    n2 += v0 * v0 + v1 * v1;
                    const int ax = n % K2, by = n / K2;
                    const bool sc = by < K && cz < K;
                    if (!(sc && ax < K)) w2 += v0 * v0;
                    if (!(sc && ax + 1 < K)) w2 += v1 * v1;
                }
            }
    }
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    if (warp == 0) tmem_dealloc(tmem_slot, C::TCOLS);
    block_sum2(n2, w2, red);
    if (tid == 0) {
        if (ch.slot < 0) {
            TR.onorm2[it.node] = n2;
            TR.ownorm2[it.node] = w2;
        }
        atomicAdd(ntrip_out, (unsigned long long)ntri);
    }
}

}  // namespace mwb
