// mw_optab.cu -- per-depth operator tables of the NS-form apply, built on the device.
//
// A convolution operator is a sum of Gaussian terms; at a depth every active term has NS matrices for the
// offsets -L .. L (mw_math.hpp, GaussianOperatorBuilder: moments, scaling blocks T, NS form), and the list
// of 3-D offsets with, per offset, the terms whose bound passes the cut (DeltaRec, TermRec).  A solver makes new
// Helmholtz operators in every iteration, so these tables are on its path: one host thread took 45 ms per
// operator (k = 8, five depths), 90 % of an iteration.  Here all operators of a batch that lack a depth are
// built together:
//   k_op_ns       one CTA per (term, offset l >= 0): four moment vectors (one warp each), three scaling
//                 blocks, F (...) F^T, and the squared norms that set the band.  Launched for l = 0 .. 3,
//                 4 .. 11 and the rest; a term whose band has ended leaves at once
//   k_op_band     one thread per term: the band's end, by the rules of the sequential construction
//   k_op_list     one thread per (term, dx, dy): counts, then writes the offsets dz above the cut
//   sorts         by bound (descending), then stably by (operator, offset): an offset's terms in decreasing order
//                 of their bounds; offsets by their largest bound
//   k_op_images   one CTA per matrix: every engine's form of it
// Latency-bound: about 0.6 ms per depth for a batch of operators (launches and four read-backs; the CTAs of
// k_op_ns take 20 us and fill the device a few times over).  Four new operators and their batched apply at k = 8:
// 189 -> 8.3 ms; the first pass of 32 new operators and trees at k = 10: 2.1 s -> 55 ms.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>

#include "mw_device.cuh"
#include "mw_kernels.cuh"
#include "mw_opplan.hpp"
#include "mw_slice.hpp"

namespace mwb {

namespace {

constexpr int kMaxBand = 4095;   // matrices of a term: offsets -L .. L with L up to this
constexpr int kMaxOffset = 511;  // listed offsets per direction up to 2 * 511 + 1 (10 bits each in the line order)

struct OpTerm {  // one (operator, term)
    double alpha, beta, cut;
    int op, m;
    int active, L;
    int base;             // first matrix of the band, within its operator
    long long row0;       // first (dx, dy) row of k_op_list
};

// whether the band of a term reaches beyond the offsets known so far (l < known), and, once it does not, its
// end; the rules of the sequential construction (t2, x2: squared norms of the s->s block and of the rest)
__device__ bool band_scan(const double* t2, const double* x2, int known, double beta, double cut, int depth, long extent,
                          int& active, int& Lout) {
    double S2 = fmax(t2[0] + x2[0], t2[1] + x2[1]);
    active = 0;
    Lout = -1;
    if (depth > 0) {
        const double xmax = sqrt(fmax(x2[0], x2[1]));
        if (beta * 10.0 * xmax * S2 < cut) return false;
    }
    long L = 1;
    while (L + 1 < extent) {
        const double last = sqrt(t2[L] + x2[L]);
        if (depth > 0 && beta * last * S2 < cut) break;
        if (depth == 0 && last <= 1e-300) break;
        if (depth == 0 && last < 1e-17 * sqrt(S2)) break;
        if (L + 1 >= known) return true;
        S2 = fmax(S2, t2[L + 1] + x2[L + 1]);
        ++L;
    }
    while (L > 0 && depth > 0 && beta * sqrt(t2[L] + x2[L]) * S2 < cut) --L;
    if (L >= extent) L = extent - 1;
    active = 1;
    Lout = (int)L;
    return false;
}

// int_0^1 Pt_p(t) exp(-a (t - c)^2) dt for p < NP by Gauss-Legendre panels graded away from the point of [0, 1]
// closest to c (unit min(a^{-1/2}, 1 / (2 a dist))); one warp, result in every lane's m[].  bp: 2 x 64 panel
// edges in shared memory
template <int NP>
__device__ void warp_moments(double a, double c, const double* px, const double* pw, int nq, double* bp, double (&m)[NP]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int p = 0; p < NP; ++p) m[p] = 0.0;
    const double cs = fmin(fmax(c, 0.0), 1.0), dist = fabs(c - cs);
    if (a * dist * dist > 800.0) return;
    int np = 0;
    if (lane == 0) {  // panels [bp[2i], bp[2i + 1]]
        if (a <= 4.0) {
            bp[0] = 0.0;
            bp[1] = 1.0;
            np = 1;
        } else {
            double u = 1.0 / sqrt(a);
            if (dist > 0.0) u = fmin(u, 1.0 / (2.0 * a * dist));
            for (int side = 0; side < 2; ++side) {
                const double sg = side ? 1.0 : -1.0, end = side ? 1.0 : 0.0;
                double prev = cs;
                for (double s = 1.0; np < 64; s *= 2.0) {
                    double b = cs + sg * s * u;
                    const bool out = side ? b >= 1.0 : b <= 0.0;
                    if (out) b = end;
                    if (b != prev) {
                        bp[2 * np] = side ? prev : b;
                        bp[2 * np + 1] = side ? b : prev;
                        ++np;
                    }
                    prev = b;
                    if (out || a * (b - c) * (b - c) > 800.0) break;
                }
            }
        }
    }
    np = __shfl_sync(0xffffffffu, np, 0);
    __syncwarp();
    for (int i = lane; i < np * nq; i += 32) {
        const int pn = i / nq, q = i - pn * nq;
        const double lo = bp[2 * pn], w = bp[2 * pn + 1] - lo;
        const double t = lo + w * px[q];
        const double g = w * pw[q] * exp(-a * (t - c) * (t - c));
        const double z = 2.0 * t - 1.0;
        double p0 = 1.0, p1 = z;
        m[0] += g;
        if (NP > 1) m[1] += g * (sqrt(3.0) * z);
#pragma unroll
        for (int p = 2; p < NP; ++p) {
            const double p2 = ((2.0 * p - 1.0) * z * p1 - (p - 1.0) * p0) * (1.0 / p);
            p0 = p1;
            p1 = p2;
            m[p] += g * (sqrt(2.0 * p + 1.0) * p2);
        }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int o = 16; o; o >>= 1) m[p] += __shfl_xor_sync(0xffffffffu, m[p], o);
    __syncwarp();
}

// NS matrix of (term, offset l) at scale n0 + depth and its norms; NS scratch block term * lcap + l
template <int K>
__global__ void __launch_bounds__(128) k_op_ns(const OpTerm* __restrict__ terms, const double* __restrict__ F,
                                               const double* __restrict__ cc, const double* __restrict__ px,
                                               const double* __restrict__ pw, int depth, int n0, long extent, int l0,
                                               int lcap, double* __restrict__ ns, double* t2, double* x2) {
    constexpr int K2 = 2 * K, KK = K * K;
    __shared__ double mom[4][K2], T[3][KK], FS[K2 * K2], A[K2 * K2], B[K2 * K2], bp[4][130], red[64];
    __shared__ int need;
    const OpTerm tm = terms[blockIdx.y];
    const int l = l0 + blockIdx.x, tid = threadIdx.x, warp = tid >> 5;
    double* t2r = t2 + (size_t)blockIdx.y * lcap;
    double* x2r = x2 + (size_t)blockIdx.y * lcap;
    if (l0 > 0) {
        if (tid == 0) {
            int act, L;
            need = band_scan(t2r, x2r, l0, tm.beta, tm.cut, depth, extent, act, L);
        }
        __syncthreads();
        if (!need) return;
    }
    const int n1 = n0 + depth + 1;  // the blocks T are those of the children's scale
    const double a = tm.alpha * ldexp(1.0, -2 * n1);
    for (int i = tid; i < K2 * K2; i += 128) FS[i] = F[i];
    {  // T(l') needs the moments about -l' and 1 - l': centres 2 - 2l, 1 - 2l, -2l, -2l - 1 for l' = 2l - 1 .. 2l + 1
        double m[K2];
        warp_moments<K2>(a, 2.0 - 2.0 * l - warp, px, pw, K2 + 20, bp[warp], m);
#pragma unroll
        for (int p = 0; p < K2; ++p)
            if ((tid & 31) == p) mom[warp][p] = m[p];
    }
    __syncthreads();
    const double fac = ldexp(1.0, -n1);
    for (int e = tid; e < KK; e += 128) {  // T(l')_ij = 2^-n sum_p c+_ijp m_p(-l') + c-_ijp m_p(1 - l')
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll 4
        for (int p = 0; p < K2; ++p) {
            const double cp = cc[p * KK + e], cm = cc[(K2 + p) * KK + e];
            s0 += cp * mom[1][p] + cm * mom[0][p];
            s1 += cp * mom[2][p] + cm * mom[1][p];
            s2 += cp * mom[3][p] + cm * mom[2][p];
        }
        T[0][e] = fac * s0;
        T[1][e] = fac * s1;
        T[2][e] = fac * s2;
    }
    __syncthreads();
    for (int e = tid; e < K2 * K2; e += 128) {  // [[T(2l) T(2l-1)]; [T(2l+1) T(2l)]]
        const int r = e / K2, c = e - r * K2, co = r >= K, ci = c >= K;
        A[e] = T[1 + co - ci][(r - co * K) * K + c - ci * K];
    }
    __syncthreads();
    for (int e = tid; e < K2 * K2; e += 128) {
        const int r = e / K2, c = e - r * K2;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < K2; ++q) s += FS[r * K2 + q] * A[q * K2 + c];
        B[e] = s;
    }
    __syncthreads();
    double tt = 0.0, xx = 0.0;
    double* out = ns + ((size_t)blockIdx.y * lcap + l) * (K2 * K2);
    for (int e = tid; e < K2 * K2; e += 128) {
        const int r = e / K2, c = e - r * K2;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < K2; ++q) s += B[r * K2 + q] * FS[c * K2 + q];
        out[e] = s;
        if (r < K && c < K) tt += s * s;
        else xx += s * s;
    }
    block_sum2(tt, xx, red);
    if (tid == 0) {
        t2r[l] = tt;
        x2r[l] = xx;
    }
}

// the terms' bands; flag[0]: some band reaches beyond lcap, flag[1]: beyond the widest supported one
__global__ void k_op_band(OpTerm* terms, int nterm, const double* t2, const double* x2, int lcap, int depth, long extent,
                          int* flag) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nterm) return;
    OpTerm& tm = terms[t];
    if (band_scan(t2 + (size_t)t * lcap, x2 + (size_t)t * lcap, lcap, tm.beta, tm.cut, depth, extent, tm.active, tm.L)) atomicOr(flag, 1);
}

__device__ __forceinline__ double bound3_dev(double beta, const double* t, const double* x, bool root) {
    if (root) return beta * sqrt((t[0] + x[0]) * (t[1] + x[1]) * (t[2] + x[2]));
    const double v = x[0] * (t[1] + x[1]) * (t[2] + x[2]) + t[0] * x[1] * (t[2] + x[2]) + t[0] * t[1] * x[2];
    return beta * sqrt(v);
}

// rows (term, dx, dy): the offsets dz whose bound reaches the cut (count, then fill at the row's place: key =
// operator | dx | dy | dz (bits each, offset by lm), bound, term).  reach: the largest listed offset, where it is wanted
__global__ void k_op_list(const OpTerm* __restrict__ terms, int nterm, long long nrows, const double* __restrict__ t2,
                          const double* __restrict__ x2, int lcap, int root, int lm, int bits, int* count,
                          const long long* __restrict__ offs, unsigned long long* key, double* bound, int* term, int* reach) {
    const long long row = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (row >= nrows) return;
    int lo = 0, hi = nterm - 1;  // last term with row0 <= row (inactive terms have no rows)
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (terms[mid].row0 <= row) lo = mid;
        else hi = mid - 1;
    }
    const OpTerm tm = terms[lo];
    const int W = 2 * tm.L + 1, q = (int)(row - tm.row0), dx = q / W - tm.L, dy = q % W - tm.L;
    const double* t2r = t2 + (size_t)lo * lcap;
    const double* x2r = x2 + (size_t)lo * lcap;
    double S2 = 0.0;
    for (int i = 0; i <= tm.L; ++i) S2 = fmax(S2, t2r[i] + x2r[i]);
    const int ix = abs(dx), iy = abs(dy);
    const double ax = t2r[ix] + x2r[ix], ay = t2r[iy] + x2r[iy];
    int n = 0, far = 0;
    const long long p0 = offs ? offs[row] : 0;
    if (root || !(tm.beta * sqrt(ax) * S2 < tm.cut || tm.beta * sqrt(ax * ay * S2) < tm.cut)) {
        for (int dz = -tm.L; dz <= tm.L; ++dz) {
            const int iz = abs(dz);
            const double t[3] = {t2r[ix], t2r[iy], t2r[iz]}, x[3] = {x2r[ix], x2r[iy], x2r[iz]};
            const double bd = bound3_dev(tm.beta, t, x, root != 0);
            if (bd <= 0.0 || bd < tm.cut) continue;
            far = max(max(ix, iy), max(far, iz));
            if (offs) {
                key[p0 + n] = ((((unsigned long long)tm.op << bits | (unsigned)(dx + lm)) << bits | (unsigned)(dy + lm)) << bits) |
                              (unsigned)(dz + lm);
                bound[p0 + n] = bd;
                term[p0 + n] = lo;
            }
            ++n;
        }
    }
    if (!offs) count[row] = n;
    if (reach && far > *reinterpret_cast<volatile int*>(reach)) atomicMax(reach, far);
}

__global__ void k_op_iota(int n, int* idx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) idx[i] = i;
}
__global__ void k_op_keys(int n, const int* __restrict__ idx, const unsigned long long* __restrict__ key,
                          unsigned long long* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = key[idx[i]];
}
__global__ void k_op_heads(int n, const unsigned long long* __restrict__ key, int* head) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) head[i] = i == 0 || key[i] != key[i - 1];
}

struct OpOut {  // one operator's lists
    TermRec* terms;
    DeltaRec* deltas;
    int rec0;  // first sorted record
    int del0;  // first offset
};
// sorted records -> TermRec; the first of each offset -> (largest bound, first record)
__global__ void k_op_terms(int n, const unsigned long long* __restrict__ key, int bits, const int* __restrict__ idx,
                           const double* __restrict__ bound, const int* __restrict__ term, const OpTerm* __restrict__ terms,
                           const int* __restrict__ head, const int* __restrict__ hpos, const OpOut* __restrict__ outs, int lm,
                           double* dmax, int* dfirst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long k = key[i];
    const unsigned mask = (1u << bits) - 1u;
    const int dz = (int)(k & mask) - lm, dy = (int)((k >> bits) & mask) - lm, dx = (int)((k >> (2 * bits)) & mask) - lm;
    const OpTerm& tm = terms[term[idx[i]]];
    const OpOut o = outs[tm.op];
    TermRec r;
    r.mx = tm.base + dx + tm.L;
    r.my = tm.base + dy + tm.L;
    r.mz = tm.base + dz + tm.L;
    r.m = tm.m;
    r.beta = tm.beta;
    r.bound = bound[idx[i]];
    o.terms[i - o.rec0] = r;
    if (head[i]) {
        dmax[hpos[i]] = r.bound;
        dfirst[hpos[i]] = i;
    }
}
__global__ void k_op_delta_keys(int n, const int* __restrict__ idx, const int* __restrict__ dfirst,
                                const unsigned long long* __restrict__ key, int bits, int* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (int)(key[dfirst[idx[i]]] >> (3 * bits));
}
// offsets in their final order: record and largest bound
__global__ void k_op_deltas(int n, const int* __restrict__ order, const int* __restrict__ dfirst, int nrec, int ndelta,
                            const unsigned long long* __restrict__ key, int bits, int lm, int reach, const double* __restrict__ dmax,
                            const OpOut* __restrict__ outs, double* maxb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int d = order[i], r0 = dfirst[d], r1 = d + 1 < ndelta ? dfirst[d + 1] : nrec;
    const unsigned long long k = key[r0];
    const unsigned mask = (1u << bits) - 1u;
    const OpOut o = outs[k >> (3 * bits)];
    DeltaRec r;
    r.d[0] = (int)((k >> (2 * bits)) & mask) - lm;
    r.d[1] = (int)((k >> bits) & mask) - lm;
    r.d[2] = (int)(k & mask) - lm;
    r.t0 = r0 - o.rec0;
    r.t1 = r1 - o.rec0;
    r.lrank = ((r.d[2] + reach) << 10) | (r.d[1] + reach);  // line order: increasing dz, then dy
    r.maxb = dmax[d];
    o.deltas[i - o.del0] = r;
    maxb[i] = r.maxb;
}

// every engine's form of a matrix (layouts: OpDepth in mw_internal.hpp, XGeo in mw_slice.hpp).  src: block of
// `blocks` and whether it is transposed (offset -l of offset l)
struct OpImages {
    double *mats, *matsD, *matsE;
    float *mats32, *matsT32, *matsbT32, *matsI, *matsbI, *matsS32, *matsbS32;
    unsigned char* matsX;
};
// FP32 -> TF32 (10 explicit mantissa bits), to nearest with ties away from zero; infinities and NaNs unchanged
__device__ __forceinline__ float tf32_round(float x) {
    unsigned u = __float_as_uint(x);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
    return __uint_as_float(u);
}
__global__ void __launch_bounds__(128) k_op_images(const int2* __restrict__ src, const double* __restrict__ blocks,
                                                   const double* __restrict__ beta, int K2, OpImages im) {
    __shared__ double M[24 * 24];
    __shared__ float sl[3][20 * 20], tl[3][10 * 10];
    const int mi = blockIdx.x, tid = threadIdx.x, n2 = K2 * K2;
    const int2 sr = src[mi];
    const double b = beta[mi];
    const double* in = blocks + (size_t)sr.x * n2;
    for (int e = tid; e < n2; e += 128) M[sr.y ? (e % K2) * K2 + e / K2 : e] = in[e];
    __syncthreads();
    const size_t at = (size_t)mi * n2;
    for (int e = tid; e < n2; e += 128) {
        im.mats[at + e] = M[e];
        im.mats32[at + e] = (float)M[e];
    }
    const int KP = (K2 + 3) / 4 * 4, RT = (K2 + 7) / 8, S = (K2 + 3) / 4, KP8 = RT * 8;
    auto val = [&](int o, int k) { return o < K2 && k < K2 ? M[o * K2 + k] : 0.0; };
    for (int e = tid; e < KP * KP; e += 128) {  // [k][o]
        const double v = val(e % KP, e / KP);
        im.matsT32[(size_t)mi * KP * KP + e] = (float)v;
        im.matsbT32[(size_t)mi * KP * KP + e] = (float)(b * v);
    }
    for (int e = tid; e < S * RT * 32; e += 128) {
        const int lane = e & 31, i = lane & 3, n = lane >> 2, q = e >> 5;
        im.matsD[(size_t)mi * S * RT * 32 + e] = val(8 * (q % RT) + n, 4 * (q / RT) + i);
        im.matsE[(size_t)mi * S * RT * 32 + e] = b * val(8 * (q / S) + 4 * (n & 1) + (n >> 1), 4 * (q % S) + i);
    }
    // three TF32 pieces (hi, mid, lo), K-major: row p KP8 + o, chunk k / 4
    for (int e = tid; e < KP8 * KP8; e += 128) {
        const int k = (e / (4 * KP8)) * 4 + e % 4, o = (e / 4) % KP8;
        for (int sc = 0; sc < 2; ++sc) {
            const double v = sc ? b * val(o, k) : val(o, k);
            const float h = tf32_round((float)v);
            const float md = tf32_round((float)(v - (double)h));
            const float lo = tf32_round((float)(v - (double)h - (double)md));
            float* img = (sc ? im.matsbI : im.matsI) + (size_t)mi * 3 * KP8 * KP8 + (size_t)(o + 3 * KP8 * (k / 4)) * 4 + k % 4;
            img[0] = h;
            img[4 * (size_t)KP8] = md;
            img[8 * (size_t)KP8] = lo;
        }
    }
    if (!im.matsX) return;
    const XGeo xg(K2);
    for (int e = tid; e < KP * KP; e += 128) {
        const int k = e / KP, o = e % KP;
        const size_t w = (size_t)mi * KP * KP + (size_t)k * KP + split_pos(o, KP / 4, 4);
        im.matsS32[w] = (float)val(o, k);
        im.matsbS32[w] = (float)(b * val(o, k));
    }
    uint16_t* img = reinterpret_cast<uint16_t*>(im.matsX + (size_t)mi * xg.OPB);
    for (int e = tid; e < xg.OPB / 4; e += 128) reinterpret_cast<uint32_t*>(img)[e] = 0u;
    if (tid < K2) slice3_row(M + tid * K2, K2, 1, sl[0] + tid * K2, sl[1] + tid * K2, sl[2] + tid * K2);
    else if (tid >= 64 && tid - 64 < xg.W2)  // the s->s block row M[o][0 .. k)
        slice3_row(M + (tid - 64) * K2, xg.W2, 1, tl[0] + (tid - 64) * xg.W2, tl[1] + (tid - 64) * xg.W2, tl[2] + (tid - 64) * xg.W2);
    __syncthreads();
    for (int e = tid; e < K2 * min(K2, 8 * xg.NCHM); e += 128) {  // (a) the operands of the data slices
        const int o = e % K2, k = e / K2;
        for (int q = 0; q < 3; ++q)
            for (int bb = q; bb < 3; ++bb) {
                uint16_t* op = img + (size_t)q * xg.OPB_Q / 2;
                op[((size_t)(k / 8) * xg.NBQ + bb * xg.W + o) * 8 + k % 8] = bf16_bits_exact(sl[bb - q][o * K2 + k]);
                if (o < xg.W2 && k < xg.W2)
                    op[((size_t)(k / 8) * xg.NBQ + xg.NCOL + bb * xg.W2 + o) * 8 + k % 8] = bf16_bits_exact(tl[bb - q][o * xg.W2 + k]);
            }
    }
    if (xg.PACK)  // (b) the packed step over x = 16 .. K2-1; data slice 3 against operator slice 0, into block 2
        for (int e = tid; e < K2 * xg.LO; e += 128) {
            const int o = e % K2, l = e / K2;
            uint16_t* pk = img + (size_t)xg.OPB_A / 2;
            for (int bb = 0; bb < 3; ++bb)
                for (int q = 0; q <= bb; ++q) {
                    const int kk = 4 * q + l;
                    pk[((size_t)(kk / 8) * xg.NCOL + bb * xg.W + o) * 8 + kk % 8] = bf16_bits_exact(sl[bb - q][o * K2 + 16 + l]);
                }
            const int kk = 12 + l;
            pk[((size_t)(kk / 8) * xg.NCOL + 2 * xg.W + o) * 8 + kk % 8] = bf16_bits_exact(sl[0][o * K2 + 16 + l]);
        }
}

template <typename T>
T* alloc(Ctx* ctx, size_t n) {
    return (T*)dalloc(ctx, sizeof(T) * std::max<size_t>(1, n));
}
int bits_for(int n) {
    int b = 1;
    while ((1 << b) < n) ++b;
    return b;
}
// (the sums have the type of `out`)
template <typename T>
void exclusive_sum(Ctx* ctx, const int* in, T* out, int n) {
    size_t tmp = 0;
    MWB_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, tmp, in, out, ::cuda::std::plus<>{}, T(0), n, ctx->stream));
    Scratch sc(ctx);
    void* d = sc.get<char>(tmp);
    MWB_CUDA(cub::DeviceScan::ExclusiveScan(d, tmp, in, out, ::cuda::std::plus<>{}, T(0), n, ctx->stream));
}
template <typename KT>
void sort_pairs(Ctx* ctx, bool descending, const KT* kin, KT* kout, const int* vin, int* vout, int n, int b0, int b1) {
    size_t tmp = 0;
    cudaStream_t s = ctx->stream;
    auto call = [&](void* d) {
        return descending ? cub::DeviceRadixSort::SortPairsDescending(d, tmp, kin, kout, vin, vout, n, b0, b1, s)
                          : cub::DeviceRadixSort::SortPairs(d, tmp, kin, kout, vin, vout, n, b0, b1, s);
    };
    MWB_CUDA(call(nullptr));
    Scratch sc(ctx);
    MWB_CUDA(call(sc.get<char>(tmp)));
}
int blocks_of(long long n, int per) { return (int)((n + per - 1) / per); }

#define MWB_OP_DISPATCH_K(k, F)                                          \
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

}  // namespace

// the matrices' images of one depth; d_src as k_op_images
void op_images(Ctx* ctx, int K2, OpDepth& od, int nmat, const int2* d_src, const double* d_blocks, const double* d_beta) {
    const int KP = (K2 + 3) / 4 * 4, RT = (K2 + 7) / 8, S = (K2 + 3) / 4, KP8 = RT * 8;
    const size_t n = (size_t)nmat;
    od.d_mats = alloc<double>(ctx, n * K2 * K2);
    od.d_mats32 = alloc<float>(ctx, n * K2 * K2);
    od.d_matsT32 = alloc<float>(ctx, n * KP * KP);
    od.d_matsbT32 = alloc<float>(ctx, n * KP * KP);
    od.d_matsD = alloc<double>(ctx, n * RT * S * 32);
    od.d_matsE = alloc<double>(ctx, n * RT * S * 32);
    od.d_matsI = alloc<float>(ctx, n * 3 * KP8 * KP8);
    od.d_matsbI = alloc<float>(ctx, n * 3 * KP8 * KP8);
    if (K2 >= 13 && K2 <= 20) {  // orders of the tensor-core x step
        const XGeo xg(K2);
        od.d_matsS32 = alloc<float>(ctx, n * KP * KP);
        od.d_matsbS32 = alloc<float>(ctx, n * KP * KP);
        od.d_matsX = alloc<unsigned char>(ctx, n * xg.OPB);
    }
    if (nmat == 0) return;
    const OpImages im{od.d_mats, od.d_matsD, od.d_matsE, od.d_mats32, od.d_matsT32, od.d_matsbT32,
                      od.d_matsI, od.d_matsbI, od.d_matsS32, od.d_matsbS32, od.d_matsX};
    k_op_images<<<nmat, 128, 0, ctx->stream>>>(d_src, d_blocks, d_beta, K2, im);
    MWB_CUDA(cudaGetLastError());
    ctx->launches++;
}

// tables of one depth for several convolution operators of one world, none of which has them yet (under its op_mtx)
static void op_build_group(const std::vector<Op*>& ops, int depth, int lcap) {
    const Mra& m = *ops[0]->mra;
    Ctx* ctx = m.ctx;
    cudaStream_t s = ctx->stream;
    const int K = m.k, K2 = 2 * K, nop = (int)ops.size();
    const bool root = depth == 0;
    long extent = 0;
    for (int d = 0; d < 3; ++d) extent = std::max<long>(extent, (long)m.boxes[d] << depth);
    // offsets 0 and 1 are always computed (the band's tests read both)
    lcap = (int)std::max<long>(2, std::min<long>(lcap, extent));
    std::vector<OpTerm> terms;
    std::vector<int> t0(nop + 1, 0);
    for (int o = 0; o < nop; ++o) {
        const double cut = root ? 0.0 : 1e-6 * ops[o]->eps * ops[o]->B0 * std::pow(4.0, -depth);
        for (size_t mi = 0; mi < ops[o]->terms.size(); ++mi)
            terms.push_back(OpTerm{ops[o]->terms[mi].alpha, ops[o]->terms[mi].beta, cut, o, (int)mi, 0, -1, 0, 0});
        t0[o + 1] = (int)terms.size();
        if (ops[o]->terms.size() > 4096) throw Error(-4, "more than 4096 operator terms");
    }
    const int nt = (int)terms.size();
    Scratch sc(ctx);
    OpTerm* d_terms = sc.up(terms);
    double* d_ns = sc.get<double>((size_t)nt * lcap * K2 * K2);
    double* d_t2 = sc.get<double>((size_t)nt * lcap);
    double* d_x2 = sc.get<double>((size_t)nt * lcap);
    int* d_flag = sc.get<int>(1);
    MWB_CUDA(cudaMemsetAsync(d_flag, 0, sizeof(int), s));
    const int cuts[4] = {0, std::min(4, lcap), std::min(12, lcap), lcap};
    for (int q = 0; q < 3; ++q) {
        if (cuts[q + 1] <= cuts[q]) continue;
        for (int y0 = 0; y0 < nt; y0 += 65535) {
            const dim3 grid(cuts[q + 1] - cuts[q], std::min(65535, nt - y0));
#define L_NS(KK)                                                                                                       \
    k_op_ns<KK><<<grid, 128, 0, s>>>(d_terms + y0, m.d_F, m.d_cc, m.d_px, m.d_pw, depth, m.n0, extent, cuts[q], lcap,  \
                                     d_ns + (size_t)y0 * lcap * K2 * K2, d_t2 + (size_t)y0 * lcap, d_x2 + (size_t)y0 * lcap);
            MWB_OP_DISPATCH_K(K, L_NS)
#undef L_NS
            MWB_CUDA(cudaGetLastError());
            ctx->launches++;
        }
    }
    if (nt > 0) {  // (an expansion whose range is empty has no terms)
        k_op_band<<<blocks_of(nt, 128), 128, 0, s>>>(d_terms, nt, d_t2, d_x2, lcap, depth, extent, d_flag);
        MWB_CUDA(cudaGetLastError());
        ctx->launches++;
    }
    int flag = 0;
    readback(ctx, {{terms.data(), d_terms, sizeof(OpTerm) * nt}, {&flag, d_flag, sizeof(int)}});
    if (root) {  // the operator scale B0, from the squared norms at l = 0
        std::vector<double> a2((size_t)nt * lcap), b2((size_t)nt * lcap);
        readback(ctx, {{a2.data(), d_t2, sizeof(double) * a2.size()}, {b2.data(), d_x2, sizeof(double) * b2.size()}});
        for (int t = 0; t < nt; ++t) {
            if (!terms[t].active) continue;
            double& B0 = ops[terms[t].op]->B0;
            B0 = std::max(B0, terms[t].beta * std::pow(a2[(size_t)t * lcap] + b2[(size_t)t * lcap], 1.5));
        }
    }
    if (flag) {  // a band wider than the scratch: once more with all of it
        sc.release();
        if (lcap > kMaxBand) throw Error(-4, "operator band wider than 8192 offsets per direction");
        for (Op* o : ops) op_build_group({o}, depth, 8 * lcap);
        return;
    }
    // bands -> matrices and list rows
    int lm = 0;
    long long nrows = 0;
    double scan = 0.0;
    std::vector<int> nmat(nop, 0);
    for (OpTerm& t : terms) {
        t.row0 = nrows;
        t.base = nmat[t.op];
        if (!t.active) continue;
        lm = std::max(lm, t.L);
        nrows += (long long)(2 * t.L + 1) * (2 * t.L + 1);
        scan += std::pow(2.0 * t.L + 1.0, 3);
        nmat[t.op] += 2 * t.L + 1;
    }
    if (lm > kMaxBand) throw Error(-4, "operator band wider than 8192 offsets per direction");
    upload_bytes(ctx, d_terms, terms.data(), sizeof(OpTerm) * nt);
    // lists
    const int bits = bits_for(2 * lm + 1), obits = bits_for(nop);
    // records per operator, counted before anything is made from them
    OpPlan plan = op_plan_rows(nop, nrows, scan);
    int* d_cnt = nullptr;
    long long* d_offs = nullptr;
    int reach = lm;  // of the lists: a wide band's, where its scaling blocks have not decayed but its bounds have, is found below
    std::vector<long long> first(nop + 1, 0);
    if (nrows > 0 && plan == OpPlan::together) {
        d_cnt = sc.get<int>(nrows + 1);
        d_offs = sc.get<long long>(nrows + 1);
        MWB_CUDA(cudaMemsetAsync(d_cnt + nrows, 0, sizeof(int), s));
        k_op_list<<<blocks_of(nrows, 128), 128, 0, s>>>(d_terms, nt, nrows, d_t2, d_x2, lcap, root, lm, bits, d_cnt, nullptr,
                                                        nullptr, nullptr, nullptr, lm > kMaxOffset ? d_flag : nullptr);
        MWB_CUDA(cudaGetLastError());
        if (lm > kMaxOffset) {
            readback(ctx, {{&reach, d_flag, sizeof(int)}});  // (zero before: no band reached beyond the scratch)
            if (reach > kMaxOffset) throw Error(-4, "operator offsets wider than 1024 per direction");
        }
        exclusive_sum(ctx, d_cnt, d_offs, (int)nrows + 1);
        // the row offsets at the operators' first terms
        std::vector<ReadReq> rq;
        for (int o = 0; o <= nop; ++o)
            rq.push_back(ReadReq{&first[o], d_offs + (t0[o] < nt ? terms[t0[o]].row0 : nrows), sizeof(long long)});
        for (size_t q = 0; q < rq.size(); q += 8) {
            auto at = [&](size_t i) { return q + i < rq.size() ? rq[q + i] : ReadReq{nullptr, nullptr, 0}; };
            readback(ctx, {at(0), at(1), at(2), at(3), at(4), at(5), at(6), at(7)});
        }
        plan = op_plan_records(nop, first[nop]);
    }
    if (plan != OpPlan::together) {
        sc.release();
        if (plan == OpPlan::refuse) throw Error(-4, "operator offset list too large");
        for (Op* o : ops) op_build_group({o}, depth, lcap);
        return;
    }
    std::vector<std::unique_ptr<OpDepth>> ods;
    for (int o = 0; o < nop; ++o) {
        ods.push_back(std::make_unique<OpDepth>(ctx));
        std::vector<int2> src;
        std::vector<double> beta;
        for (int t = t0[o]; t < t0[o + 1]; ++t)
            for (int l = -terms[t].L; terms[t].active && l <= terms[t].L; ++l) {
                src.push_back(int2{t * lcap + std::abs(l), l < 0 ? 1 : 0});
                beta.push_back(terms[t].beta);
            }
        Scratch lists(ctx);
        const int2* d_src = lists.up(src);
        op_images(ctx, K2, *ods[o], nmat[o], d_src, d_ns, lists.up(beta));
    }
    std::vector<int> rec0(first.begin(), first.end()), del0(nop + 1, 0);
    std::vector<double> maxb;
    if (nrows > 0) {
        const int nrec = rec0[nop];
        const int rb = blocks_of(nrec, 256);
        if (nrec > 0) {
            auto* d_key = sc.get<unsigned long long>(nrec);
            auto* d_key2 = sc.get<unsigned long long>(nrec);
            auto* d_key3 = sc.get<unsigned long long>(nrec);
            double* d_bound = sc.get<double>(nrec);
            double* d_b2 = sc.get<double>(nrec);
            int* d_term = sc.get<int>(nrec);
            int* d_i0 = sc.get<int>(nrec);
            int* d_i1 = sc.get<int>(nrec);
            int* d_head = sc.get<int>(nrec + 1);
            int* d_hpos = sc.get<int>(nrec + 1);
            k_op_list<<<blocks_of(nrows, 128), 128, 0, s>>>(d_terms, nt, nrows, d_t2, d_x2, lcap, root, lm, bits, d_cnt, d_offs,
                                                            d_key, d_bound, d_term, nullptr);
            k_op_iota<<<rb, 256, 0, s>>>(nrec, d_i0);
            sort_pairs(ctx, true, reinterpret_cast<const unsigned long long*>(d_bound), reinterpret_cast<unsigned long long*>(d_b2),
                       d_i0, d_i1, nrec, 0, 64);
            k_op_keys<<<rb, 256, 0, s>>>(nrec, d_i1, d_key, d_key2);
            sort_pairs(ctx, false, d_key2, d_key3, d_i1, d_i0, nrec, 0, 3 * bits + obits);
            MWB_CUDA(cudaMemsetAsync(d_head + nrec, 0, sizeof(int), s));
            k_op_heads<<<rb, 256, 0, s>>>(nrec, d_key3, d_head);
            exclusive_sum(ctx, d_head, d_hpos, nrec + 1);
            {
                std::vector<ReadReq> rq;
                for (int o = 0; o <= nop; ++o) rq.push_back(ReadReq{&del0[o], d_hpos + rec0[o], sizeof(int)});
                for (size_t q = 0; q < rq.size(); q += 8) {
                    auto at = [&](size_t i) { return q + i < rq.size() ? rq[q + i] : ReadReq{nullptr, nullptr, 0}; };
                    readback(ctx, {at(0), at(1), at(2), at(3), at(4), at(5), at(6), at(7)});
                }
            }
            const int nd = del0[nop], db = blocks_of(nd, 256);
            std::vector<OpOut> outs(nop);
            for (int o = 0; o < nop; ++o) {
                ods[o]->d_terms = alloc<TermRec>(ctx, rec0[o + 1] - rec0[o]);
                ods[o]->d_deltas = alloc<DeltaRec>(ctx, del0[o + 1] - del0[o]);
                outs[o] = OpOut{ods[o]->d_terms, ods[o]->d_deltas, rec0[o], del0[o]};
            }
            OpOut* d_outs = sc.up(outs);
            double* d_dmax = sc.get<double>(nd);
            double* d_dm2 = sc.get<double>(nd);
            double* d_maxb = sc.get<double>(nd);
            int* d_df = sc.get<int>(nd);
            int* d_o0 = sc.get<int>(nd);
            int* d_o1 = sc.get<int>(nd);
            int* d_k0 = sc.get<int>(nd);
            int* d_k1 = sc.get<int>(nd);
            k_op_terms<<<rb, 256, 0, s>>>(nrec, d_key3, bits, d_i0, d_bound, d_term, d_terms, d_head, d_hpos, d_outs, lm, d_dmax, d_df);
            k_op_iota<<<db, 256, 0, s>>>(nd, d_o0);
            sort_pairs(ctx, true, reinterpret_cast<const unsigned long long*>(d_dmax), reinterpret_cast<unsigned long long*>(d_dm2),
                       d_o0, d_o1, nd, 0, 64);
            if (nop > 1) {
                k_op_delta_keys<<<db, 256, 0, s>>>(nd, d_o1, d_df, d_key3, bits, d_k0);
                sort_pairs(ctx, false, d_k0, d_k1, d_o1, d_o0, nd, 0, obits);
                std::swap(d_o0, d_o1);
            }
            k_op_deltas<<<db, 256, 0, s>>>(nd, d_o1, d_df, nrec, nd, d_key3, bits, lm, reach, d_dmax, d_outs, d_maxb);
            MWB_CUDA(cudaGetLastError());
            ctx->launches += 9;
            maxb.resize(nd);
            readback(ctx, {{maxb.data(), d_maxb, sizeof(double) * nd}});
        }
    }
    for (int o = 0; o < nop; ++o) {
        OpDepth& od = *ods[o];
        if (!od.d_terms) od.d_terms = alloc<TermRec>(ctx, 0);
        if (!od.d_deltas) od.d_deltas = alloc<DeltaRec>(ctx, 0);
        for (int t = t0[o]; t < t0[o + 1]; ++t) {
            od.base.push_back(terms[t].base);
            od.band.push_back(terms[t].active ? terms[t].L : -1);
        }
        od.maxb.assign(maxb.begin() + del0[o], maxb.begin() + del0[o + 1]);
        ops[o]->depths.emplace(depth, std::move(ods[o]));
    }
}

void op_build_tables(const std::vector<Op*>& ops, int depth) {
    // at most eight operators at a time: bounds the matrices' scratch (8 x 134 terms x 64 offsets x 4.6 KB at k = 12);
    // that of the lists is bounded by the plan
    for (size_t q = 0; q < ops.size(); q += 8)
        op_build_group(std::vector<Op*>(ops.begin() + q, ops.begin() + std::min(ops.size(), q + 8)), depth, 64);
}

}  // namespace mwb
