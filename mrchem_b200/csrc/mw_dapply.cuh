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
// register-tiled scalar GEMM reads 10 shared words per 25 FMAs and ran at the shared-memory rate.  Contraction
// time of whole applies, scalar kernel -> this one: 16 Helmholtz orbitals at k = 10 46.2 -> 25.4 ms (the
// instructions alone, padded rows included: 17.8), 20-atom Poisson at k = 12 302 -> 41.2 ms (37.3), three-charge
// Poisson at k = 8, prec 1e-5 5.1 -> 2.1 ms, at k = 6 3.11 -> 1.19 ms (prec 1e-5) and 1.44 -> 0.58 (prec 1e-3).
//
// Work split (k = 6 and k > 8 share the last pairs out as extra units, see DCfg).  Warp p owns the z-index pair
// (c = p, p + k): one slice of the scaling half and one of the wavelet half, so that generated (scaling-only) inputs and the s->s correction load every warp alike.
// The x product of its 2 x 2k columns (b, c) accumulates in registers over the line's triples (rows a',
// columns b: the FP64 C fragment), and that fragment is the A operand of the y product as it stands: a
// lane's two C values are columns 2j and 2j+1, so with columns ordered b = 8t + 4e + j (e the parity) each
// of the two values is one A fragment of four consecutive b.  Nothing is exchanged between warps, no
// barrier is needed, until a plane's y sums go to shared memory (T2) for the z product.  When 2k mod 8 is
// 2 or 4 the two slices share one column tile (even columns one slice, odd columns the other): at k = 10
// the pair's 40 columns are exactly five tiles.  Rows are padded to a multiple of 8 (2k = 20: 24).
//
// Staging.  Each warp streams its own columns of the triples' block images (fragment order, one slab per
// step of four a) through a private ring of NS slots by cp.async: no two warps wait for one another.  The
// order of slabs is fixed (S per triple, NS divides S), so slot and refill of every step are compile-time
// constants; a run-time list of slabs with the operators among them cost 580 cycles of dependent integer work
// per step against 340 of products, and bulk copies issued by one lane 100 to 240 cycles.  The operators'
// fragments are read from global memory (L1 / L2 hits: every warp reads the same) one step ahead of the
// products that use them, as are the slabs' fragments.
//
// Below the root the s->s block (T x T x T on the scaling part) is left out: the steps a < k of the
// corner tiles (a', b < k of the scaling slice) accumulate apart (S), are added to the full sums at the
// line's end, and go through their own y product into U2; the z product takes U2 off with -Tz as further
// steps of the same accumulators.  FP64 accumulators of the output block live in tensor memory between
// planes (one read and one write per plane).
#pragma once

namespace mwb {

template <int K>
struct DCfg {
    static constexpr int K2 = 2 * K;
    static constexpr int RT = (K2 + 7) / 8;   // row tiles of an operator
    static constexpr int S = (K2 + 3) / 4;    // steps of a contraction over 2k
    static constexpr int FT = K2 / 8, REM = K2 % 8;
    static constexpr int WOFF = FT + (REM != 0 ? 1 : 0);               // first own tile of the wavelet slice
    static constexpr int NTP = 2 * FT + (REM == 0 ? 0 : REM <= 4 ? 1 : 2);  // column tiles of a pair
    // one pair per warp; at k = 6 and from k = 9 up fewer: eight warps (two per SM sub-partition, 255 registers each) take a pair
    // each and share the last K - 8 pairs by slices: an extra unit = one slice c, at most one per warp.  (One warp
    // per pair puts three warps on one or two sub-partitions and two on the others at k = 9, 10.)  k = 6 likewise
    // with four warps of a pair and an extra unit each: 1.33 -> 1.23 ms in a three-charge Poisson apply at prec 1e-5; at k = 5 the two extra
    // units leave two warps idle for a third of the time (1.13 -> 1.16, not used).
    static constexpr int NWARP = K > 8 ? 8 : K == 6 ? 4 : K, NTHR = 32 * NWARP;
    static constexpr int NXU = 2 * (K - NWARP);  // extra units: pair 8 + u / 2, slice u mod 2
    static constexpr bool XU = NXU > 0;
    static constexpr int RS = (K + 7) / 8;    // row and column tiles of the scaling corner
    static constexpr int KS = (K + 3) / 4;    // steps of a contraction over k
    static constexpr bool MIXED = K % 4 != 0; // the last of them also covers wavelet indices
    static constexpr int SLABX = NTP * 32, SLABU = XU ? RT * 32 : 0, SLAB = SLABX + SLABU;  // a slab: the pair's and the extra unit's columns
    static constexpr int MATD = S * RT * 32;           // operator image
    static constexpr int IMG = NWARP * S * SLABX + NXU * S * SLABU;  // block image: every warp's slabs (pair, extra unit)
    __host__ __device__ static constexpr int img_off(int w) { return S * (w * SLABX + (w < NXU ? w : NXU) * SLABU); }
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
    static constexpr int MAXT = 128;  // triples per chunk whose records are kept in shared memory
    static constexpr int MINB = K <= 4 ? 4 : K <= 5 ? 3 : K <= 8 ? 2 : 1;
    static constexpr int FIXED = 8 * (K2 * LD2 + K * LDU) + MAXT * 16;
    static constexpr int BUDGET = 232448 / MINB - 2048 - 1024;  // less the static part and the reserved part
    static constexpr int NS_FIT = (BUDGET - FIXED) / (8 * NWARP * SLAB);
    // ring slots: a triple's slabs; two triples' where a slab's products are too few to cover the latency of the
    // slabs behind it (k <= 6); half a triple's where shared memory ends (k = 12)
    static constexpr int NS = K <= 6 ? 2 * S : NS_FIT >= S ? S : S / 2;
    static constexpr bool TWO = NS == 2 * S;
    static constexpr size_t SMEM = FIXED + (size_t)8 * NWARP * NS * SLAB;
    static_assert(NS <= NS_FIT && NS >= 2 && (TWO || S % NS == 0) && NXU <= NWARP && TCOLS_NEED <= 512 && MINB * TCOLS <= 512 && RS <= FT && RS <= 2, "DCfg");
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

// Block images of the FP64 engine, in the order the x step's B fragments are read: [warp][step s][pair's tiles,
// extra unit's tiles], a slab's tiles as [tile couple][lane][2], then a last odd tile [lane]; lane = 4 n + i holds
// X[a = 4s + i][column n] (an extra unit's tiles: eight b each).  One CTA per block; the four lanes of a column read one 32-byte sector, writes are contiguous.  Slot numbering as
// k_ximage; a generated node's block is its k^3 scaling part.  Bound by HBM (one read, one write).
template <int K>
__global__ void __launch_bounds__(256) k_dimage(const ImgSrc* __restrict__ srcs, int nsrc, const double* __restrict__ gblk,
                                                long long nreal, double* __restrict__ img) {
    using C = DCfg<K>;
    constexpr int K2 = C::K2;
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
    auto value = [&](int s, int bb, int sl, int p) -> double {
        const int a = 4 * s + i, c = sl ? p + K : p;
        if (real) return a < K2 && bb < K2 ? b[a + K2 * (bb + K2 * c)] : 0.0;
        return a < K && bb < K && !sl ? b[a + K * (bb + K * c)] : 0.0;
    };
    auto slab = [&](double* o, auto ntiles, auto&& tile) {
        constexpr int NT = decltype(ntiles)::value;
#pragma unroll
        for (int q = 0; q < NT / 2; ++q)
            *reinterpret_cast<double2*>(o + 64 * q + 2 * lane) = make_double2(tile(2 * q), tile(2 * q + 1));
        if constexpr (NT % 2 != 0) o[32 * (NT - 1) + lane] = tile(NT - 1);
    };
    for (int ps = warp; ps < C::NWARP * C::S; ps += 8) {
        const int p = ps / C::S, s = ps - p * C::S;
        double* o = out + C::img_off(p) + s * (p < C::NXU ? C::SLAB : C::SLABX);
        slab(o, std::integral_constant<int, C::NTP>(), [&](int j) { return value(s, dcol_b<K>(j, n), dcol_slice<K>(j, n), p); });
        if (p < C::NXU)
            slab(o + C::SLABX, std::integral_constant<int, C::RT>(),
                 [&](int j) { return value(s, 8 * j + 4 * (n & 1) + (n >> 1), p & 1, C::NWARP + p / 2); });
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
    const double* __restrict__ mats = TR.matsD;   // A fragments (x, z)
    const double* __restrict__ matsy = TR.matsE;  // beta-scaled B fragments (y)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fi = lane & 3, fn = lane >> 2;  // fragment coordinates: A (row fn, k fi), B (k fi, column fn)
    const int ntri = ch.c1 - ch.c0;
    const int zw = C::NWARP - 1 - warp;  // z tiles zw + NWARP q: the odd ones go to warps without an extra unit

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

    // ---- staging: slab s of a triple goes to slot s % NS (TWO: of its half of the ring), one commit group per slab
    const bool hasx = C::XU && warp < C::NXU;                 // extra unit: slice xc, of the scaling half or not
    const bool xs = hasx && (warp & 1) == 0;
    const int xp = C::NWARP + warp / 2, xc = xp + K * (warp & 1);
    double* ring = ring0 + (size_t)warp * NS * SLAB;
    const int off = C::img_off(warp) + 2 * lane;
    auto image = [&](const DTri& h) { return dimg + (size_t)h.slot * C::IMG + off; };
    auto issue = [&](double* to, const double* px, int s, auto hx) {  // px: this lane's place in a triple's image
        constexpr int SL = decltype(hx)::value ? SLAB : C::SLABX;
        double* dst = to + 2 * lane;
#pragma unroll
        for (int e = 0; e < SL; e += 64)
            if (e + 64 <= SL || lane < (SL - e) / 2) cp_async16(dst + e, px + s * SL + e);
    };
    auto frag = [&](const double* tab, int mi, int q) { return __ldg(tab + (size_t)mi * C::MATD + q * 32 + lane); };

    double D[RT][NTP][2];                       // x sums of the line (of the corner: the steps a >= k)
    double SC[RS][RS][2];                       // ... of the corner: the steps a < k
    double DX[RT][RT][2], SX[RS][RS][2];        // the same of the extra unit (columns b = 8 j + 4 e + fi of its slice)
    double anext[RT];                           // x operator fragments of the next triple's first step
    // one x step: fragments, and their products.  PART 0: a < k, 1: both halves (k no multiple of 4), 2: a >= k;
    // HX: with the extra unit; GEN: generated input (columns in the first RS tiles only, a < k)
    struct Frag {
        double a[RT], b[NTP + 1], bx[C::XU ? RT + 1 : 1];
    };
    auto load_tiles = [&](const double* q, double* b, auto ntiles, auto nload) {
        constexpr int NT = decltype(ntiles)::value;
#pragma unroll
        for (int j = 0; j < decltype(nload)::value; j += 2) {
            if (j + 1 < NT) {
                const double2 v = *reinterpret_cast<const double2*>(q + 32 * j + 2 * lane);
                b[j] = v.x;
                b[j + 1] = v.y;
            } else {
                b[j] = q[32 * j + lane];
            }
        }
    };
    auto xmul = [&](const Frag& f, const int PART, auto hx, auto gen) {
        constexpr bool HX = decltype(hx)::value, GEN = decltype(gen)::value;
        const bool low = PART == 0 || (PART == 1 && 4 * (KS - 1) + fi < K);
#pragma unroll
        for (int j = 0; j < (GEN ? RS : NTP); ++j)
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                if (j < RS && r < RS) {
                    if (PART <= 1) dmma(SC[r][j], low ? f.a[r] : 0.0, f.b[j]);
                    if (!GEN && PART >= 1) dmma(D[r][j], low ? 0.0 : f.a[r], f.b[j]);
                } else {
                    dmma(D[r][j], f.a[r], f.b[j]);
                }
            }
        if constexpr (HX) {
#pragma unroll
            for (int j = 0; j < (GEN ? RS : RT); ++j)
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    if (j < RS && r < RS) {
                        if (PART <= 1) dmma(SX[r][j], low ? f.a[r] : 0.0, f.bx[j]);
                        if (!GEN && PART >= 1) dmma(DX[r][j], low ? 0.0 : f.a[r], f.bx[j]);
                    } else {
                        dmma(DX[r][j], f.a[r], f.bx[j]);
                    }
                }
        }
    };
    // the fragments of slab s
    auto xload = [&](Frag& f, const double* rp, int s, auto hx, auto gen) {
        constexpr bool HX = decltype(hx)::value, GEN = decltype(gen)::value;
        const double* sx = rp + (s % NS) * SLAB;
        if (!GEN || s < KS) {  // a generated input is zero beyond
            load_tiles(sx, f.b, std::integral_constant<int, NTP>(), std::integral_constant<int, GEN ? RS : NTP>());
            if constexpr (HX)
                load_tiles(sx + C::SLABX, f.bx, std::integral_constant<int, RT>(), std::integral_constant<int, GEN ? RS : RT>());
        }
    };
    // x product of the chunk's i-th triple: D[a'][(b, c)] += sum_a Mx[a'][a] X[a][(b, c)]; hn, hm: the next two
    // (within the chunk).  On entry slab 0 has landed for every lane, on exit the next triple's
    auto xtriple = [&](int i, const DTri& h, const DTri& hn, const DTri& hm, auto hx, auto gen) {
        constexpr bool GEN = decltype(gen)::value;
        double* rp = ring + (C::TWO ? (i & 1) * S * SLAB : 0);        // the triple's slots
        double* rq = ring + (C::TWO ? ((i & 1) ^ 1) * S * SLAB : 0);  // its neighbours'
        const double *p0 = image(h), *p1 = image(hn), *p2 = image(hm);
        Frag f[2];
#pragma unroll
        for (int r = 0; r < RT; ++r) f[0].a[r] = anext[r];
        xload(f[0], rp, 0, hx, gen);
#pragma unroll
        for (int s = 0; s < S; ++s) {
            // every lane read slab s - 1 before the previous step's barrier: its slot takes the slab NS further on
            const int n = s - 1 + NS;
            double* to = (C::TWO && s == 0 ? rq : rp) + ((s - 1 + S) % (C::TWO ? S : NS)) * SLAB;
            if (n < S) issue(to, p0, n, hx);
            else if (n < 2 * S && i + 1 < ntri) issue(to, p1, n - S, hx);
            else if (n >= 2 * S && i + 2 < ntri) issue(to, p2, n - 2 * S, hx);
            cp_async_commit();
            cp_async_wait_group<NS - 2>();
            __syncwarp();  // slab s + 1 is in for every lane
            if (s + 1 < S) {
#pragma unroll
                for (int r = 0; r < RT; ++r) f[(s + 1) & 1].a[r] = frag(mats, h.mx, (s + 1) * RT + r);
                xload(f[(s + 1) & 1], rp, s + 1, hx, gen);
            } else {
#pragma unroll
                for (int r = 0; r < RT; ++r) anext[r] = frag(mats, hn.mx, r);
            }
            if (!GEN || s < KS) xmul(f[s & 1], s >= KS ? 2 : (C::MIXED && s == KS - 1) ? 1 : 0, hx, gen);
        }
    };
    // y: T2[c][a'][b'] (+)= sum_b D[a'][b] beta My[b'][b] for column tile j of b' (a plane sums its lines), and
    // the s->s block U2[c][a'][b'] (+)= sum_{b<k} SC[a'][b] beta Ty[b'][b]
    // m: the operator's fragments of this tile; replaced by those of tile j + 1
    auto ycol = [&](int j, int my, bool first_line, auto hx, double* mj) {
        constexpr bool HX = decltype(hx)::value;
        double m[S];
#pragma unroll
        for (int s = 0; s < S; ++s) m[s] = mj[s];
        if (j + 1 < RT) {
#pragma unroll
            for (int s = 0; s < S; ++s) mj[s] = frag(matsy, my, (j + 1) * S + s);
        }
        const bool corr = j < RS && !root;
        double Y[2][RT][2], Z[RS][2];
        [[maybe_unused]] double YX[RT][2], ZX[RS][2];  // the extra unit's
        const int b0 = 8 * j + fi;
        auto t2at = [&](int c, int a8) { return T2 + c * LD2 + a8 + fn + PP * b0; };
        // value at (row a8 + fn, b' = b0 + 4 e): the plane's sum so far, or zero
        auto prev = [&](const double* p, int a8, int e, int lim) {
            return !first_line && a8 + fn < lim && b0 + 4 * e < lim ? p[4 * e * PP] : 0.0;
        };
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int sl = 0; sl < 2; ++sl) Y[sl][r][e] = prev(t2at(warp + sl * K, 8 * r), 8 * r, e, K2);
#pragma unroll
            for (int r = 0; r < RS; ++r) Z[r][e] = prev(U2 + warp * LDU + 8 * r + fn + PP * b0, 8 * r, e, K);
            if constexpr (HX) {
#pragma unroll
                for (int r = 0; r < RT; ++r) YX[r][e] = prev(t2at(xc, 8 * r), 8 * r, e, K2);
#pragma unroll
                for (int r = 0; r < RS; ++r) ZX[r][e] = xs ? prev(U2 + xp * LDU + 8 * r + fn + PP * b0, 8 * r, e, K) : 0.0;
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            // step s = 2 t + e of a slice: parity e of its tile t, or its parity of the shared tile
            constexpr bool SH = C::REM != 0 && C::REM <= 4;
            const int e0 = (SH && s == 2 * FT) ? 0 : s % 2, e1 = (SH && s == 2 * FT) ? 1 : s % 2;
            const int t0 = (SH && s == 2 * FT) ? FT : s / 2, t1 = (SH && s == 2 * FT) ? FT : C::WOFF + s / 2;
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                dmma(Y[0][r], D[r][t0][e0], m[s]);
                dmma(Y[1][r], D[r][t1][e1], m[s]);
            }
            if constexpr (HX) {
#pragma unroll
                for (int r = 0; r < RT; ++r) dmma(YX[r], DX[r][s / 2][s % 2], m[s]);
            }
        }
        if (corr) {
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                const double mc = 4 * s + fi < K ? m[s] : 0.0;
#pragma unroll
                for (int r = 0; r < RS; ++r) dmma(Z[r], SC[r][s / 2][s % 2], mc);
                if constexpr (HX)
                    if (xs) {
#pragma unroll
                        for (int r = 0; r < RS; ++r) dmma(ZX[r], SX[r][s / 2][s % 2], mc);
                    }
            }
        }
        auto put = [&](double* p, int a8, int e, int lim, double v) {
            if (a8 + fn < lim && b0 + 4 * e < lim) p[4 * e * PP] = v;
        };
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
            for (int r = 0; r < RT; ++r) {
#pragma unroll
                for (int sl = 0; sl < 2; ++sl) put(t2at(warp + sl * K, 8 * r), 8 * r, e, K2, Y[sl][r][e]);
                if constexpr (HX) put(t2at(xc, 8 * r), 8 * r, e, K2, YX[r][e]);
            }
            if (corr) {
#pragma unroll
                for (int r = 0; r < RS; ++r) {
                    put(U2 + warp * LDU + 8 * r + fn + PP * b0, 8 * r, e, K, Z[r][e]);
                    if constexpr (HX)
                        if (xs) put(U2 + xp * LDU + 8 * r + fn + PP * b0, 8 * r, e, K, ZX[r][e]);
                }
            }
        }
    };
    // z: acc[c'][(a', b')] += sum_c Mz[c'][c] T2[c][(a', b')]  - the s->s block
    auto zplane = [&](int mz, const double* a0) {  // a0: the operator's fragments of step 0
        uint32_t w[2 * C::ZD];
        tmem_span_ld<0, 2 * C::ZD>(tacc, w);
        tmem_span_wait<0, 2 * C::ZD>(w);
        double z[ZT][RT][2];
#pragma unroll
        for (int q = 0; q < C::ZD; ++q) z[q / (2 * RT)][(q / 2) % RT][q % 2] = words_to_double(w[2 * q], w[2 * q + 1]);
        double a[2][RT], b[2][ZT];
        const bool last = C::NZT % C::NWARP == 0 || zw + C::NWARP * (ZT - 1) < C::NZT;  // the warp's last tile exists
        auto load = [&](int f, int s) {
#pragma unroll
            for (int r = 0; r < RT; ++r) a[f][r] = s == 0 ? a0[r] : frag(mats, mz, s * RT + r);
            const int c = 4 * s + fi;
#pragma unroll
            for (int q = 0; q < ZT; ++q)
                b[f][q] = (4 * s + 3 < K2 || c < K2) && (q + 1 < ZT || last)
                              ? T2[c * LD2 + C::phys(8 * (zw + C::NWARP * q)) + fn] : 0.0;
        };
        load(0, 0);
        static_for<S>([&](auto SI) {
            constexpr int s = decltype(SI)::value, f = s & 1;
            if constexpr (s + 1 < S) load(f ^ 1, s + 1);
#pragma unroll
            for (int q = 0; q < ZT; ++q)
                if (q + 1 < ZT || last) {
#pragma unroll
                    for (int r = 0; r < RT; ++r) dmma(z[q][r], a[f][r], b[f][q]);
                }
            if constexpr (s < KS)
                if (!root) {
                    const int c = 4 * s + fi;
                    double ac[RS];
#pragma unroll
                    for (int r = 0; r < RS; ++r) ac[r] = (8 * r + fn < K && c < K) ? -a[f][r] : 0.0;
#pragma unroll
                    for (int q = 0; q < ZT; ++q) {
                        const int n0 = 8 * (zw + C::NWARP * q);  // columns with some a', b' < k
                        if (n0 < K * K2 && (n0 % K2 < K || n0 % K2 + 7 >= K2)) {
                            const double bu = c < K ? U2[c * LDU + C::phys(n0) + fn] : 0.0;
#pragma unroll
                            for (int r = 0; r < RS; ++r) dmma(z[q][r], ac[r], bu);
                        }
                    }
                }
        });
#pragma unroll
        for (int q = 0; q < C::ZD; ++q) double_to_words(z[q / (2 * RT)][(q / 2) % RT][q % 2], w[2 * q], w[2 * q + 1]);
        tmem_span_st<0, 2 * C::ZD>(tacc, w);
        tmem_wait_st();
    };
    using Yes = std::true_type;
    using No = std::false_type;
    using WithX = std::integral_constant<bool, C::XU>;
    DTri hn{}, hm{};
    if (ntri > 0) {
        hn = rec(ch.c0);
        hm = rec(ch.c0 + min(1, ntri - 1));
#pragma unroll
        for (int s = 0; s + 1 < NS; ++s) {
            if (s < S || ntri > 1) {
                const double* px = image(s < S ? hn : hm);
                if (C::XU && hasx) issue(ring + s * SLAB, px, s % S, WithX());
                else issue(ring + s * SLAB, px, s % S, No());
            }
            cp_async_commit();
        }
#pragma unroll
        for (int r = 0; r < RT; ++r) anext[r] = frag(mats, hn.mx, r);
        cp_async_wait_group<NS - 2>();
        __syncwarp();
    }
    for (int i = 0; i < ntri;) {  // planes (a chunk ends with a plane, a plane with a line)
        bool first_line = true;
        DTri h;
        do {  // lines
#pragma unroll
            for (int r = 0; r < RT; ++r) {
#pragma unroll
                for (int j = 0; j < NTP; ++j) D[r][j][0] = D[r][j][1] = 0.0;
#pragma unroll
                for (int j = 0; j < RT; ++j) DX[r][j][0] = DX[r][j][1] = 0.0;
            }
#pragma unroll
            for (int r = 0; r < RS; ++r)
#pragma unroll
                for (int j = 0; j < RS; ++j) SC[r][j][0] = SC[r][j][1] = SX[r][j][0] = SX[r][j][1] = 0.0;
            do {
                h = hn;
                hn = hm;
                hm = rec(ch.c0 + min(i + 2, ntri - 1));
                if (C::XU && hasx) {
                    if (h.flags & DT_GEN) xtriple(i, h, hn, hm, WithX(), Yes());
                    else xtriple(i, h, hn, hm, WithX(), No());
                } else {
                    if (h.flags & DT_GEN) xtriple(i, h, hn, hm, No(), Yes());
                    else xtriple(i, h, hn, hm, No(), No());
                }
                ++i;
            } while (!(h.flags & DT_LEND));
            double mj[S];
#pragma unroll
            for (int s = 0; s < S; ++s) mj[s] = frag(matsy, h.my, s);
            if (first_line) __syncthreads();  // the previous plane's z step has read T2 and U2
#pragma unroll
            for (int j = 0; j < RS; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int r = 0; r < RS; ++r) {
                        D[r][j][e] += SC[r][j][e];
                        DX[r][j][e] += SX[r][j][e];
                    }
#pragma unroll 1
            for (int j = 0; j < RT; ++j) {
                if (C::XU && hasx) ycol(j, h.my, first_line, WithX(), mj);
                else ycol(j, h.my, first_line, No(), mj);
            }
            first_line = false;
        } while (!(h.flags & DT_PEND));
        double a0[RT];
#pragma unroll
        for (int r = 0; r < RT; ++r) a0[r] = frag(mats, (int)h.mz, r);
        __syncthreads();  // the plane's y sums are in T2, U2
        zplane((int)h.mz, a0);
    }
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
                const int cz = 8 * r + fn, n = 8 * (zw + C::NWARP * q) + 2 * fi;
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
