// Kernel templates instantiated once per quartet class and variant by the
// generated translation units (gen_eri.py).  One warp owns one work item and
// evaluates one quartet per lane and step: a row item holds 32 ket pairs, one
// per lane, against the bra pairs of one second shell in turn (plain builds), a
// pair item one bra pair against a run of ket pairs (density-screened and
// multi-density builds, the ERI tensor).  Work items are pulled from a
// per-launch queue head with atomicAdd, so the grid is persistent (sized to the
// resident capacity of the SMs).
#pragma once

#include "vlx_device.cuh"

namespace vlx {

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of N values (N <= 32) over the warp by recursive halving: at each level
// a lane hands half of its values to its partner and keeps the other half, so
// that N values cost about N + 5 exchanges instead of the 5 N of N separate
// warp sums.  On return v[0] of a lane is the sum of element `e` (one lane
// for each e in [0, N); e < 0: nothing).
template <int N, int O, typename T>
__device__ __forceinline__ void warp_sums_level(T* v, const int lane, int& e, int& cnt, bool& own)
{
    if constexpr (O > 0) {
        const bool up = (lane & O) != 0;
        if constexpr (N > 1) {
            constexpr int H = (N + 1) / 2;
#pragma unroll
            for (int k = 0; k < H; k++) {
                const T lo = v[k], hi = (k + H < N) ? v[k + H] : T(0);
                v[k] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, O);
            }
            e += up ? H : 0;
            cnt = up ? max(cnt - H, 0) : min(cnt, H);
            warp_sums_level<H, O / 2>(v, lane, e, cnt, own);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            own = own && !up;
            warp_sums_level<1, O / 2>(v, lane, e, cnt, own);
        }
    }
}

template <int N, typename T>
__device__ __forceinline__ int warp_sums(T* v, const int lane)
{
    int e = 0, cnt = N;
    bool own = true;
    warp_sums_level<N, 16>(v, lane, e, cnt, own);
    return (own && cnt > 0) ? e : -1;
}

template <typename T>
__device__ __forceinline__ T ldD(const T* __restrict__ D, int nao, int r, int c)
{
    return __ldg(D + (size_t)r * nao + c);
}

template <typename T>
__device__ __forceinline__ void addF(T* F, int nao, int r, int c, T v)
{
    red_add(F + (size_t)r * nao + c, v);
}

// J/K digestion of the spherical block f[((i NB + j) NC + k) ND + l] of one
// unique shell quartet (P Q | R S).  s carries the permutational weight
// (1/2 for P == Q, 1/2 for R == S, 1/2 for PQ == RS) and is 0 on idle lanes.
// Symmetric density (reference local_distribute_rest_*): contributions are
// accumulated in one orientation and the caller adds the transpose at the end.
// T = double, or float for the FP32 digestion of FP32 quartets into the
// separate FP32 accumulator of a density-screened build (FP32 copy of D).
template <int NA, int NB, int NC, int ND, int MODE, typename T>
__device__ __forceinline__ void digest_t(const T* f, const T s, const int lane, const int p0, const int nlp,
                                         const int q0, const int nlq, const int r0, const int nlr, const int s0,
                                         const int nls, const T* __restrict__ D, T* F, const int nao, const T cjw,
                                         const T ckw)
{
    const T cj = cjw * s, ck = ckw * s;
    if (cjw != T(0)) {
        // F_PQ: reduce over the lanes (ket pairs), then one atomic per element
#pragma unroll
        for (int i = 0; i < NA; i++) {
#pragma unroll
            for (int j = 0; j < NB; j++) {
                T v = T(0);
#pragma unroll
                for (int k = 0; k < NC; k++) {
#pragma unroll
                    for (int l = 0; l < ND; l++) {
                        T d = ldD(D, nao, r0 + k * nlr, s0 + l * nls);
                        if (MODE == MODE_FOCK_GEN) d += ldD(D, nao, s0 + l * nls, r0 + k * nlr);
                        v = fma(f[((i * NB + j) * NC + k) * ND + l], d, v);
                    }
                }
                v = warp_sum(v * cj);
                if (lane == ((i * NB + j) & 31)) {
                    addF(F, nao, p0 + i * nlp, q0 + j * nlq, v);
                    if (MODE == MODE_FOCK_GEN) addF(F, nao, q0 + j * nlq, p0 + i * nlp, v);
                }
            }
        }
        // F_RS: per lane
        if (s != T(0)) {
#pragma unroll
            for (int k = 0; k < NC; k++) {
#pragma unroll
                for (int l = 0; l < ND; l++) {
                    T v = T(0);
#pragma unroll
                    for (int i = 0; i < NA; i++) {
#pragma unroll
                        for (int j = 0; j < NB; j++) {
                            T d = ldD(D, nao, p0 + i * nlp, q0 + j * nlq);
                            if (MODE == MODE_FOCK_GEN) d += ldD(D, nao, q0 + j * nlq, p0 + i * nlp);
                            v = fma(f[((i * NB + j) * NC + k) * ND + l], d, v);
                        }
                    }
                    addF(F, nao, r0 + k * nlr, s0 + l * nls, cj * v);
                    if (MODE == MODE_FOCK_GEN) addF(F, nao, s0 + l * nls, r0 + k * nlr, cj * v);
                }
            }
        }
    }
    if (ckw != T(0) && s != T(0)) {
        // F_PR += sum_{j l} f D_QS ; F_RP (general) += sum f D_SQ
#pragma unroll
        for (int i = 0; i < NA; i++) {
#pragma unroll
            for (int k = 0; k < NC; k++) {
                T v = T(0), w = T(0);
#pragma unroll
                for (int j = 0; j < NB; j++) {
#pragma unroll
                    for (int l = 0; l < ND; l++) {
                        const T x = f[((i * NB + j) * NC + k) * ND + l];
                        v = fma(x, ldD(D, nao, q0 + j * nlq, s0 + l * nls), v);
                        if (MODE == MODE_FOCK_GEN) w = fma(x, ldD(D, nao, s0 + l * nls, q0 + j * nlq), w);
                    }
                }
                addF(F, nao, p0 + i * nlp, r0 + k * nlr, ck * v);
                if (MODE == MODE_FOCK_GEN) addF(F, nao, r0 + k * nlr, p0 + i * nlp, ck * w);
            }
        }
        // F_PS += sum_{j k} f D_QR
#pragma unroll
        for (int i = 0; i < NA; i++) {
#pragma unroll
            for (int l = 0; l < ND; l++) {
                T v = T(0), w = T(0);
#pragma unroll
                for (int j = 0; j < NB; j++) {
#pragma unroll
                    for (int k = 0; k < NC; k++) {
                        const T x = f[((i * NB + j) * NC + k) * ND + l];
                        v = fma(x, ldD(D, nao, q0 + j * nlq, r0 + k * nlr), v);
                        if (MODE == MODE_FOCK_GEN) w = fma(x, ldD(D, nao, r0 + k * nlr, q0 + j * nlq), w);
                    }
                }
                addF(F, nao, p0 + i * nlp, s0 + l * nls, ck * v);
                if (MODE == MODE_FOCK_GEN) addF(F, nao, s0 + l * nls, p0 + i * nlp, ck * w);
            }
        }
        // F_QR += sum_{i l} f D_PS
#pragma unroll
        for (int j = 0; j < NB; j++) {
#pragma unroll
            for (int k = 0; k < NC; k++) {
                T v = T(0), w = T(0);
#pragma unroll
                for (int i = 0; i < NA; i++) {
#pragma unroll
                    for (int l = 0; l < ND; l++) {
                        const T x = f[((i * NB + j) * NC + k) * ND + l];
                        v = fma(x, ldD(D, nao, p0 + i * nlp, s0 + l * nls), v);
                        if (MODE == MODE_FOCK_GEN) w = fma(x, ldD(D, nao, s0 + l * nls, p0 + i * nlp), w);
                    }
                }
                addF(F, nao, q0 + j * nlq, r0 + k * nlr, ck * v);
                if (MODE == MODE_FOCK_GEN) addF(F, nao, r0 + k * nlr, q0 + j * nlq, ck * w);
            }
        }
        // F_QS += sum_{i k} f D_PR
#pragma unroll
        for (int j = 0; j < NB; j++) {
#pragma unroll
            for (int l = 0; l < ND; l++) {
                T v = T(0), w = T(0);
#pragma unroll
                for (int i = 0; i < NA; i++) {
#pragma unroll
                    for (int k = 0; k < NC; k++) {
                        const T x = f[((i * NB + j) * NC + k) * ND + l];
                        v = fma(x, ldD(D, nao, p0 + i * nlp, r0 + k * nlr), v);
                        if (MODE == MODE_FOCK_GEN) w = fma(x, ldD(D, nao, r0 + k * nlr, p0 + i * nlp), w);
                    }
                }
                addF(F, nao, q0 + j * nlq, s0 + l * nls, ck * v);
                if (MODE == MODE_FOCK_GEN) addF(F, nao, s0 + l * nls, q0 + j * nlq, ck * w);
            }
        }
    }
}

template <int NA, int NB, int NC, int ND, int MODE>
__device__ __forceinline__ void digest(const double* f, const double s, const int lane, const int p0, const int nlp,
                                       const int q0, const int nlq, const int r0, const int nlr, const int s0,
                                       const int nls, const MolDev& m, const double cjw, const double ckw)
{
    digest_t<NA, NB, NC, ND, MODE, double>(f, s, lane, p0, nlp, q0, nlq, r0, nlr, s0, nls, m.D, m.F, m.nao, cjw, ckw);
}

// ---- row items: the lanes keep their ket pair RS and the bra pairs PQ of one
// second shell Q pass by, so the terms that do not involve P stay with the
// lane: F_QR, F_QS and F_RS are summed in `acc` over the item and added to F
// once (flush_row), and the elements D_QR, D_QS, D_RS are read once into `dc`.
// Per step remain the gathers of D_PR and D_PS, the additions to F_PR and
// F_PS, and one warp reduction of F_PQ: for (sp|ss) 2 gathers and 2 reductions
// per quartet where digesting each quartet by itself takes 8 and 9.  The s, p
// and d classes of the (H2O)32 / def2-SVP build take 34 ms in all with, 49 ms
// without these sums; (sp|ss) 7.55 -> 5.7 ms, then bound by FP64 and instruction
// issue (FP64 pipe 46%, issue 57% of the cycles).
// Layout of both: [QR: NB NC | QS: NB ND | RS: NC ND], and for a general
// density (GEN) the transposes of the first two [RQ | SQ] behind; RS then
// stands for both orientations (D_RS + D_SR, equal additions).
// acc is the lane's column of a per-warp shared-memory array (element stride
// kColumn), dc another or, with DS = 1 for its stride, registers.
constexpr int kColumn = 32;

template <int NB, int NC, int ND, bool GEN>
struct RowLayout {
    static constexpr int QS = NB * NC, RS = QS + NB * ND, T = RS + NC * ND, N = GEN ? T + RS : T;
};

template <bool TR>
__device__ __forceinline__ double ldT(const MolDev& m, const int r, const int c)
{
    return TR ? ldD(m.D, m.nao, c, r) : ldD(m.D, m.nao, r, c);
}

template <bool TR>
__device__ __forceinline__ void addT(const MolDev& m, const int r, const int c, const double v)
{
    if (TR)
        addF(m.F, m.nao, c, r, v);
    else
        addF(m.F, m.nao, r, c, v);
}

// The AO indices of component 0 and the component strides of the four shells.
struct QuartetAO {
    int p0, q0, r0, s0, nlp, nlq, nlr, nls;
    __device__ __forceinline__ int p(int i) const { return p0 + i * nlp; }
    __device__ __forceinline__ int q(int j) const { return q0 + j * nlq; }
    __device__ __forceinline__ int r(int k) const { return r0 + k * nlr; }
    __device__ __forceinline__ int s(int l) const { return s0 + l * nls; }
};

// Exchange part of one step; TR: the transposed elements of a general density.
template <int NA, int NB, int NC, int ND, bool TR, int DS>
__device__ __forceinline__ void digest_row_k(const double* f, const double ck, const QuartetAO& o, const MolDev& m,
                                             double* acc, const double* dc)
{
    using L = RowLayout<NB, NC, ND, TR>;
    constexpr int base = TR ? L::T : 0;
    {
        double d[NA * ND];
#pragma unroll
        for (int i = 0; i < NA; i++)
#pragma unroll
            for (int l = 0; l < ND; l++) d[i * ND + l] = ck * ldT<TR>(m, o.p(i), o.s(l));
#pragma unroll
        for (int j = 0; j < NB; j++)
#pragma unroll
            for (int k = 0; k < NC; k++) {
                double x = acc[kColumn * (base + j * NC + k)];
#pragma unroll
                for (int i = 0; i < NA; i++)
#pragma unroll
                    for (int l = 0; l < ND; l++) x = fma(f[((i * NB + j) * NC + k) * ND + l], d[i * ND + l], x);
                acc[kColumn * (base + j * NC + k)] = x;
            }
    }
    {
        double d[NA * NC];
#pragma unroll
        for (int i = 0; i < NA; i++)
#pragma unroll
            for (int k = 0; k < NC; k++) d[i * NC + k] = ck * ldT<TR>(m, o.p(i), o.r(k));
#pragma unroll
        for (int j = 0; j < NB; j++)
#pragma unroll
            for (int l = 0; l < ND; l++) {
                double x = acc[kColumn * (base + L::QS + j * ND + l)];
#pragma unroll
                for (int i = 0; i < NA; i++)
#pragma unroll
                    for (int k = 0; k < NC; k++) x = fma(f[((i * NB + j) * NC + k) * ND + l], d[i * NC + k], x);
                acc[kColumn * (base + L::QS + j * ND + l)] = x;
            }
    }
    {
        double x[NA * NC];
#pragma unroll
        for (int e = 0; e < NA * NC; e++) x[e] = 0.0;
#pragma unroll
        for (int j = 0; j < NB; j++)
#pragma unroll
            for (int l = 0; l < ND; l++) {
                const double d = dc[DS * (base + L::QS + j * ND + l)];
#pragma unroll
                for (int i = 0; i < NA; i++)
#pragma unroll
                    for (int k = 0; k < NC; k++)
                        x[i * NC + k] = fma(f[((i * NB + j) * NC + k) * ND + l], d, x[i * NC + k]);
            }
        if (ck != 0.0) {
#pragma unroll
            for (int i = 0; i < NA; i++)
#pragma unroll
                for (int k = 0; k < NC; k++) addT<TR>(m, o.p(i), o.r(k), ck * x[i * NC + k]);
        }
    }
    {
        double x[NA * ND];
#pragma unroll
        for (int e = 0; e < NA * ND; e++) x[e] = 0.0;
#pragma unroll
        for (int j = 0; j < NB; j++)
#pragma unroll
            for (int k = 0; k < NC; k++) {
                const double d = dc[DS * (base + j * NC + k)];
#pragma unroll
                for (int i = 0; i < NA; i++)
#pragma unroll
                    for (int l = 0; l < ND; l++)
                        x[i * ND + l] = fma(f[((i * NB + j) * NC + k) * ND + l], d, x[i * ND + l]);
            }
        if (ck != 0.0) {
#pragma unroll
            for (int i = 0; i < NA; i++)
#pragma unroll
                for (int l = 0; l < ND; l++) addT<TR>(m, o.p(i), o.s(l), ck * x[i * ND + l]);
        }
    }
}

// s: the permutational weight of the lane's quartet, 0 on an idle lane.
template <int NA, int NB, int NC, int ND, bool GEN, int DS>
__device__ __forceinline__ void digest_row(const double* f, const double s, const int lane, const QuartetAO& o,
                                           const MolDev& m, const double cjw, const double ckw, double* acc,
                                           const double* dc)
{
    using L = RowLayout<NB, NC, ND, GEN>;
    if (cjw != 0.0) {
        const double cj = cjw * s;
        double d[NC * ND > NA * NB ? NC * ND : NA * NB];
#pragma unroll
        for (int k = 0; k < NC; k++)
#pragma unroll
            for (int l = 0; l < ND; l++) d[k * ND + l] = cj * dc[DS * (L::RS + k * ND + l)];
        // F_PQ: chunks of up to 32 elements, each reduced over the lanes
        constexpr int NPQ = NA * NB, NCH = (NPQ + 31) / 32, CH = (NPQ + NCH - 1) / NCH;
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            double v[CH];
#pragma unroll
            for (int e = 0; e < CH; e++) {
                v[e] = 0.0;
                if (c * CH + e < NPQ) {
#pragma unroll
                    for (int kl = 0; kl < NC * ND; kl++) v[e] = fma(f[(c * CH + e) * NC * ND + kl], d[kl], v[e]);
                }
            }
            const int e = warp_sums<CH>(v, lane) + c * CH;
            if (e >= c * CH && e < NPQ) {
                addF(m.F, m.nao, o.p(e / NB), o.q(e % NB), v[0]);
                if (GEN) addF(m.F, m.nao, o.q(e % NB), o.p(e / NB), v[0]);
            }
        }
        // F_RS
#pragma unroll
        for (int i = 0; i < NA; i++)
#pragma unroll
            for (int j = 0; j < NB; j++) {
                double x = ldD(m.D, m.nao, o.p(i), o.q(j));
                if (GEN) x += ldD(m.D, m.nao, o.q(j), o.p(i));
                d[i * NB + j] = cj * x;
            }
#pragma unroll
        for (int kl = 0; kl < NC * ND; kl++) {
            double x = acc[kColumn * (L::RS + kl)];
#pragma unroll
            for (int ij = 0; ij < NA * NB; ij++) x = fma(f[ij * NC * ND + kl], d[ij], x);
            acc[kColumn * (L::RS + kl)] = x;
        }
    }
    if (ckw != 0.0) {
        digest_row_k<NA, NB, NC, ND, false, DS>(f, ckw * s, o, m, acc, dc);
        if (GEN) digest_row_k<NA, NB, NC, ND, true, DS>(f, ckw * s, o, m, acc, dc);
    }
}

// Start of a row item: clears the lane's accumulators and reads its elements
// of D (the lanes without a ket pair read a valid one's).
template <int NB, int NC, int ND, bool TR, int DS>
__device__ __forceinline__ void read_row_k(const QuartetAO& o, const MolDev& m, double* dc)
{
    using L = RowLayout<NB, NC, ND, TR>;
    constexpr int base = TR ? L::T : 0;
#pragma unroll
    for (int j = 0; j < NB; j++) {
#pragma unroll
        for (int k = 0; k < NC; k++) dc[DS * (base + j * NC + k)] = ldT<TR>(m, o.q(j), o.r(k));
#pragma unroll
        for (int l = 0; l < ND; l++) dc[DS * (base + L::QS + j * ND + l)] = ldT<TR>(m, o.q(j), o.s(l));
    }
}

template <int NB, int NC, int ND, bool GEN, int DS>
__device__ __forceinline__ void begin_row(const QuartetAO& o, const MolDev& m, const double cj, const double ck,
                                          double* acc, double* dc)
{
    using L = RowLayout<NB, NC, ND, GEN>;
#pragma unroll
    for (int e = 0; e < L::N; e++) acc[kColumn * e] = 0.0;
    if (ck != 0.0) {
        read_row_k<NB, NC, ND, false, DS>(o, m, dc);
        if (GEN) read_row_k<NB, NC, ND, true, DS>(o, m, dc);
    }
    if (cj != 0.0) {
#pragma unroll
        for (int k = 0; k < NC; k++)
#pragma unroll
            for (int l = 0; l < ND; l++) {
                double x = ldD(m.D, m.nao, o.r(k), o.s(l));
                if (GEN) x += ldD(m.D, m.nao, o.s(l), o.r(k));
                dc[DS * (L::RS + k * ND + l)] = x;
            }
    }
}

// End of a row item: the lane's accumulators into F.
template <int NB, int NC, int ND, bool TR>
__device__ __forceinline__ void flush_row_k(const QuartetAO& o, const MolDev& m, const double* acc)
{
    using L = RowLayout<NB, NC, ND, TR>;
    constexpr int base = TR ? L::T : 0;
#pragma unroll
    for (int j = 0; j < NB; j++) {
#pragma unroll
        for (int k = 0; k < NC; k++) addT<TR>(m, o.q(j), o.r(k), acc[kColumn * (base + j * NC + k)]);
#pragma unroll
        for (int l = 0; l < ND; l++) addT<TR>(m, o.q(j), o.s(l), acc[kColumn * (base + L::QS + j * ND + l)]);
    }
}

template <int NB, int NC, int ND, bool GEN>
__device__ __forceinline__ void flush_row(const QuartetAO& o, const MolDev& m, const double cj, const double ck,
                                          const double* acc)
{
    using L = RowLayout<NB, NC, ND, GEN>;
    if (ck != 0.0) {
        flush_row_k<NB, NC, ND, false>(o, m, acc);
        if (GEN) flush_row_k<NB, NC, ND, true>(o, m, acc);
    }
    if (cj != 0.0) {
#pragma unroll
        for (int k = 0; k < NC; k++)
#pragma unroll
            for (int l = 0; l < ND; l++) {
                const double v = acc[kColumn * (L::RS + k * ND + l)];
                addF(m.F, m.nao, o.r(k), o.s(l), v);
                if (GEN) addF(m.F, m.nao, o.s(l), o.r(k), v);
            }
    }
}

// Scatter one unique spherical quartet into the dense ERI tensor (all eight
// index permutations), as CT4CEriTensorDistributor does.
template <int NA, int NB, int NC, int ND>
__device__ __forceinline__ void scatter_eri(const double* f, const int p0, const int nlp, const int q0, const int nlq,
                                            const int r0, const int nlr, const int s0, const int nls, double* eri,
                                            const int nao)
{
    const size_t n = (size_t)nao;
    for (int i = 0; i < NA; i++)
        for (int j = 0; j < NB; j++)
            for (int k = 0; k < NC; k++)
                for (int l = 0; l < ND; l++) {
                    const size_t p = p0 + i * nlp, q = q0 + j * nlq, r = r0 + k * nlr, t = s0 + l * nls;
                    const double v = f[((i * NB + j) * NC + k) * ND + l];
                    eri[((p * n + q) * n + r) * n + t] = v;
                    eri[((q * n + p) * n + r) * n + t] = v;
                    eri[((p * n + q) * n + t) * n + r] = v;
                    eri[((q * n + p) * n + t) * n + r] = v;
                    eri[((r * n + t) * n + p) * n + q] = v;
                    eri[((t * n + r) * n + p) * n + q] = v;
                    eri[((r * n + t) * n + q) * n + p] = v;
                    eri[((t * n + r) * n + q) * n + p] = v;
                }
}

constexpr int kWarpsPerBlock = 4;

// Per-class tuning traits, specialised in each class's generated unit from the
// tables of gen_eri.py (BLOCKS_HINT, STAGE_BRA, row_sums), so that tuning one
// class recompiles only that unit:
//   BlocksHint::value  minimum resident 128-thread blocks per SM the register
//                      allocation of a kernel variant must allow (0: no minimum);
//   StageBra::value    the pair-item kernel stages the bra primitive records
//                      in shared memory per work item (PairViewS);
//   RowStore::sums     the row-item kernels keep an item's accumulators and
//                      elements of D in per-warp shared-memory arrays
//                      (digest_row), ::d_registers the latter in registers;
//                      without sums every step is digested by itself;
//   RowStore::stream   a step's integrals go through StreamSink.
template <int LA, int LB, int LC, int LD, int V>
struct BlocksHint;
template <int LA, int LB, int LC, int LD>
struct StageBra;
template <int LA, int LB, int LC, int LD, bool GEN>
struct RowStore;

// The Boys coefficients of the one order a class needs (the lower orders
// follow by recursion), staged once per persistent block: the per-lane table
// lookups then gather from shared memory instead of L1/L2.
template <typename R>
constexpr int boys_stride = sizeof(R) == sizeof(float) ? BOYS_STRIDE_F : BOYS_STRIDE;

template <int L, typename R>
__device__ __forceinline__ void stage_boys(const FockArgs& a, R* sboys)
{
    const R* tab;
    if constexpr (sizeof(R) == sizeof(float))
        tab = a.boys_f;
    else
        tab = a.boys;
    for (int i = threadIdx.x; i < boys_stride<R>; i += blockDim.x) sboys[i] = __ldg(tab + L * boys_stride<R> + i);
    __syncthreads();
}

// Takes a quartet's integrals into the array f[((i NB + j) NC + k) ND + l].
template <int NAB, int NC, int ND, typename R>
struct ArraySink {
    R* f;
    template <int K, int L>
    __device__ __forceinline__ void put(const R* o)
    {
#pragma unroll
        for (int ij = 0; ij < NAB; ij++) f[(ij * NC + K) * ND + L] = o[ij];
    }
};

// The class's integrals of one quartet, in FP64 or FP32 by the type of the
// Boys table, into a sink.
template <class C, class Bra, class Ket, class Sink>
__device__ __forceinline__ void eri_compute(const Bra& bra, const Ket& ket, const double* tab, const double omega2,
                                            Sink& sink)
{
    C::compute(bra, ket, tab, omega2, sink);
}
template <class C, class Bra, class Ket, class Sink>
__device__ __forceinline__ void eri_compute(const Bra& bra, const Ket& ket, const float* tab, const double omega2,
                                            Sink& sink)
{
    C::compute_f32(bra, ket, tab, (float)omega2, sink);
}

// J/K digestion of one quartet (symmetric density) as its integrals arrive, one
// ket component (k, l) at a time: the classes whose block f does not fit the
// registers (up to 49 x 49 values) need no array of it, which a lane would
// write once and read six times through thread-local memory ((pf|pd) of the
// (H2O)27 / def2-TZVP build 15.0 -> 12.4 ms, (pd|pd) 7.5 -> 6.4, the build
// 246 -> 237).
// s: the permutational weight, 0 on an idle lane.
template <int NA, int NB, int NC, int ND, typename R>
struct StreamSink {
    const QuartetAO& o;
    const MolDev& m;
    const double cj, ck;  // weights of the label times s
    const bool j_on, k_on;
    double pq[NA * NB], qr[NB], pr[NA], qs[NB * ND], ps[NA * ND];

    __device__ __forceinline__ StreamSink(const QuartetAO& ao, const MolDev& mol, const double cjw, const double ckw,
                                          const double s)
        : o(ao), m(mol), cj(cjw * s), ck(ckw * s), j_on(cjw != 0.0), k_on(ckw != 0.0)
    {
#pragma unroll
        for (int e = 0; e < NA * NB; e++) pq[e] = 0.0;
#pragma unroll
        for (int e = 0; e < NB * ND; e++) qs[e] = 0.0;
#pragma unroll
        for (int e = 0; e < NA * ND; e++) ps[e] = 0.0;
    }

    template <int K, int L>
    __device__ __forceinline__ void put(const R* f)
    {
        if (j_on) {
            const double d = cj * ldD(m.D, m.nao, o.r(K), o.s(L));
            double x = 0.0;
#pragma unroll
            for (int i = 0; i < NA; i++)
#pragma unroll
                for (int j = 0; j < NB; j++) {
                    const double v = (double)f[i * NB + j];
                    pq[i * NB + j] = fma(v, d, pq[i * NB + j]);
                    x = fma(v, ldD(m.D, m.nao, o.p(i), o.q(j)), x);
                }
            if (cj != 0.0) addF(m.F, m.nao, o.r(K), o.s(L), cj * x);
        }
        if (k_on) {
            if (L == 0) {
#pragma unroll
                for (int j = 0; j < NB; j++) qr[j] = 0.0;
#pragma unroll
                for (int i = 0; i < NA; i++) pr[i] = 0.0;
            }
            double dqr[NB], dqs[NB];
#pragma unroll
            for (int j = 0; j < NB; j++) {
                dqr[j] = ldD(m.D, m.nao, o.q(j), o.r(K));
                dqs[j] = ldD(m.D, m.nao, o.q(j), o.s(L));
            }
#pragma unroll
            for (int i = 0; i < NA; i++) {
                const double dpr = ldD(m.D, m.nao, o.p(i), o.r(K)), dps = ldD(m.D, m.nao, o.p(i), o.s(L));
#pragma unroll
                for (int j = 0; j < NB; j++) {
                    const double v = (double)f[i * NB + j];
                    qr[j] = fma(v, dps, qr[j]);
                    pr[i] = fma(v, dqs[j], pr[i]);
                    qs[j * ND + L] = fma(v, dpr, qs[j * ND + L]);
                    ps[i * ND + L] = fma(v, dqr[j], ps[i * ND + L]);
                }
            }
            if (ck != 0.0) {
                if (L == ND - 1) {
#pragma unroll
                    for (int j = 0; j < NB; j++) addF(m.F, m.nao, o.q(j), o.r(K), ck * qr[j]);
#pragma unroll
                    for (int i = 0; i < NA; i++) addF(m.F, m.nao, o.p(i), o.r(K), ck * pr[i]);
                }
                if (K == NC - 1) {
#pragma unroll
                    for (int j = 0; j < NB; j++) addF(m.F, m.nao, o.q(j), o.s(L), ck * qs[j * ND + L]);
#pragma unroll
                    for (int i = 0; i < NA; i++) addF(m.F, m.nao, o.p(i), o.s(L), ck * ps[i * ND + L]);
                }
            }
        }
    }

    // F_PQ over the lanes (all lanes of the warp)
    __device__ __forceinline__ void finish(const int lane)
    {
        if (!j_on) return;
        constexpr int NPQ = NA * NB, NCH = (NPQ + 31) / 32, CH = (NPQ + NCH - 1) / NCH;
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            double v[CH];
#pragma unroll
            for (int e = 0; e < CH; e++) v[e] = (c * CH + e < NPQ) ? pq[c * CH + e] : 0.0;
            const int e = warp_sums<CH>(v, lane) + c * CH;
            if (e >= c * CH && e < NPQ) addF(m.F, m.nao, o.p(e / NB), o.q(e % NB), v[0]);
        }
    }
};
__device__ __forceinline__ PairView make_view(const PairBlockDev& b, int i, int kuse, double)
{
    return {b.prim + prim_offset(b.kprim, i), b.ab + ab_offset(i), kuse};
}
__device__ __forceinline__ PairViewF make_view(const PairBlockDev& b, int i, int kuse, float)
{
    return {b.primf + prim_offset(b.kprim, i), b.abf + ab_offset(i), kuse};
}
__device__ __forceinline__ PairViewR<double> make_row_view(const PairBlockDev& b, int q, int kuse, double)
{
    return {b.rprim + (size_t)q * b.kprim * 10, b.rab + 4 * (size_t)q, kuse};
}
__device__ __forceinline__ PairViewR<float> make_row_view(const PairBlockDev& b, int q, int kuse, float)
{
    return {b.rprimf + (size_t)q * b.kprim * 10, b.rabf + 4 * (size_t)q, kuse};
}

// One step of a work item: lane evaluates ket pair jj of kb against the bra
// pair (act = false: an idle lane, which computes and contributes nothing)
// and digests the spherical block.
// With the per-quartet density screening, multi-density digestion and the
// device quartet counters; the plain builds take row_body.
template <int LA, int LB, int LC, int LD, bool GEN, typename R>
__device__ __forceinline__ void quartet_step(const FockArgs& a, const int mode, const int lane,
                                             const PairBlockDev& bb, const PairBlockDev& kb, const int bbi,
                                             const int kbi, const WorkItem& w, const PairViewT<R>& bra,
                                             const MolDev& m, const int p0, const int q0, const double s_bra,
                                             const int jj, const bool act, const R* sboys, const R* sbra)
{
    using C = EriClass<LA, LB, LC, LD>;
    constexpr bool f32 = sizeof(R) == sizeof(float);
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1, NC = 2 * LC + 1, ND = 2 * LD + 1;
    const int nlp = m.nl[LA], nlq = m.nl[LB], nlr = m.nl[LC], nls = m.nl[LD];
    const PairViewT<R> ket = make_view(kb, jj, __ldg(kb.nuse + jj), R());
    if (a.qstat) {
        const unsigned n = __popc(__ballot_sync(0xffffffffu, act));
        const unsigned pq = __reduce_add_sync(0xffffffffu, act ? (unsigned)(bra.kuse * ket.kuse) : 0u);
        if (lane == 0) {
            atomicAdd(a.qstat, (unsigned long long)n);
            atomicAdd(a.qstat + 1, (unsigned long long)pq);
        }
    }
    R g[C::NSPH];
    ArraySink<NA * NB, NC, ND, R> sink{g};
    if (StageBra<LA, LB, LC, LD>::value && sbra) {
        PairViewS<R> bs;
        bs.s = sbra;
        bs.ab = bra.ab;
        bs.kuse = bra.kuse;
        eri_compute<C>(bs, ket, sboys, a.omega2, sink);
    } else {
        eri_compute<C>(bra, ket, sboys, a.omega2, sink);
    }
    if constexpr (f32) {
        // density-screened build with an FP32 accumulator: the FP32 quartets
        // (each contribution below the FP32 cutoff) are digested in FP32
        // against the FP32 copy of D
        if (a.F32 != nullptr && (mode & 3) != MODE_ERI) {
            const int r0 = __ldg(kb.ao + jj), s0 = __ldg(kb.ao + kb.npairs + jj);
            float s = act ? (float)s_bra : 0.0f;
            if (r0 == s0) s *= 0.5f;
            if (bbi == kbi && jj == w.bra) s *= 0.5f;
            digest_t<NA, NB, NC, ND, GEN ? MODE_FOCK_GEN : MODE_FOCK_SYM, float>(
                g, s, lane, p0, nlp, q0, nlq, r0, nlr, s0, nls, a.D32, a.F32, m.nao, (float)a.cj, (float)a.ck);
            return;
        }
    }
    double f[C::NSPH];
#pragma unroll
    for (int t = 0; t < C::NSPH; t++) f[t] = (double)g[t];
    const int r0 = __ldg(kb.ao + jj), s0 = __ldg(kb.ao + kb.npairs + jj);
    if (GEN && (mode & 3) == MODE_ERI) {
        if (act) scatter_eri<NA, NB, NC, ND>(f, p0, nlp, q0, nlq, r0, nlr, s0, nls, a.eri, m.nao);
    } else {
        double s = act ? s_bra : 0.0;
        if (r0 == s0) s *= 0.5;
        if (bbi == kbi && jj == w.bra) s *= 0.5;
        // one density, or each density of a multi-density build in turn
        const int nd = a.dens.n > 0 ? a.dens.n : 1;
#pragma unroll 1
        for (int d = 0; d < nd; d++) {
            MolDev md = m;
            double cj = a.cj, ck = a.ck;
            if (a.dens.n > 0) {
                md.D = a.dens.D[d];
                md.F = a.dens.F[d];
                cj = a.dens.cj[d];
                ck = a.dens.ck[d];
            }
            digest<NA, NB, NC, ND, GEN ? MODE_FOCK_GEN : MODE_FOCK_SYM>(f, s, lane, p0, nlp, q0, nlq, r0, nlr, s0, nls,
                                                                        md, cj, ck);
        }
    }
}

// Pair items.
template <int LA, int LB, int LC, int LD, bool GEN, typename R>
__device__ __forceinline__ void quartet_body(const FockArgs& a, const int mode)
{
    constexpr bool f32 = sizeof(R) == sizeof(float);
    const int lane = threadIdx.x & 31;
    __shared__ __align__(16) R sboys[boys_stride<R>];
    // per warp: the staged bra primitive records of the current work item
    __shared__ __align__(16) R sbra_all[StageBra<LA, LB, LC, LD>::value ? kWarpsPerBlock * kStageBraMax * 10 : 2];
    stage_boys<LA + LB + LC + LD>(a, sboys);
    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(a.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= a.nitems) return;
        const WorkItem w = a.items[it];
        const int bbi = w.blocks & 0xffff, kbi = (unsigned)w.blocks >> 16;
        const PairBlockDev bb = a.blocks[bbi];
        const PairBlockDev kb = a.blocks[kbi];
        const MolDev m = a.mols ? a.mols[bb.mol] : a.mol;
        const PairViewT<R> bra = make_view(bb, w.bra, __ldg(bb.nuse + w.bra), R());
        const int p0 = __ldg(bb.ao + w.bra), q0 = __ldg(bb.ao + bb.npairs + w.bra);
        const double s_bra = (p0 == q0) ? 0.5 : 1.0;
        const R* sbra = nullptr;
        if constexpr (StageBra<LA, LB, LC, LD>::value) {
            if (bra.kuse <= kStageBraMax) {
                R* s = sbra_all + (threadIdx.x >> 5) * kStageBraMax * 10;
                __syncwarp();  // the previous item's reads are done
                stage_bra(s, bra, lane);
                __syncwarp();
                sbra = s;
            }
        }
        int k0, k1;
        // per warp: kets that passed the density screening, waiting for a full step
        __shared__ int squeue[kWarpsPerBlock][64];
        int* queue = squeue[threadIdx.x >> 5];
        // with density screening the precision is decided per quartet below,
        // so both launches walk the item's whole ket range
        item_range(a, bb, kb, w, f32 && !a.dsh, k0, k1);
        int P = 0, Q = 0;
        float qpq = 0.0f, dpq = 0.0f;
        if (a.dsh) {
            P = __ldg(bb.sh + w.bra);
            Q = __ldg(bb.sh + bb.npairs + w.bra);
            qpq = __ldg(bb.q + w.bra);
            dpq = __ldg(a.dsh + (size_t)P * a.nsh + Q);
            k1 = density_ket_end(a, P, Q, qpq, dpq, kb, f32, k1);
        }
        // steps of 32 kets; with density screening the kets this launch keeps
        // are first compacted into full steps (order preserved)
        int n = 0, j0 = k0;
        for (;;) {
            int jj;
            bool act;
            if (!a.dsh) {
                if (j0 >= k1) break;
                const int j = j0 + lane;
                act = j < k1;
                jj = act ? j : (k1 - 1);
                j0 += 32;
            } else {
                while (n < 32 && j0 < k1) {
                    const int j = j0 + lane;
                    const bool keep = (j < k1) && quartet_kept(a, quartet_bound(a, P, Q, qpq, dpq, kb, j), f32);
                    const unsigned mask = __ballot_sync(0xffffffffu, keep);
                    if (keep) queue[n + __popc(mask & ((1u << lane) - 1u))] = j;
                    n += __popc(mask);
                    j0 += 32;
                    __syncwarp();
                }
                if (n == 0) break;
                act = lane < n;
                jj = queue[act ? lane : 0];
                __syncwarp();
                if (lane < n - 32) queue[lane] = queue[lane + 32];
                n = max(n - 32, 0);
                __syncwarp();
            }
            quartet_step<LA, LB, LC, LD, GEN, R>(a, mode, lane, bb, kb, bbi, kbi, w, bra, m, p0, q0, s_bra, jj, act, sboys,
                                         sbra);
        }
    }
}

// Row items (plain builds): lane j holds ket pair kbeg + j for the whole item
// and the bra pairs of one second shell Q pass by (see digest_row).
// Dynamic shared memory: the Boys order, then the accumulators and elements of
// D that RowStore keeps there.
template <int LA, int LB, int LC, int LD, bool GEN>
constexpr int row_elements = RowLayout<2 * LB + 1, 2 * LC + 1, 2 * LD + 1, GEN>::N;

template <int LA, int LB, int LC, int LD, bool GEN, typename R>
constexpr int row_shared_bytes()
{
    using Store = RowStore<LA, LB, LC, LD, GEN>;
    return (boys_stride<R> * (int)sizeof(R) + 15) / 16 * 16 +
           (Store::sums + (Store::sums && !Store::d_registers)) * kWarpsPerBlock * kColumn *
               row_elements<LA, LB, LC, LD, GEN> * 8;
}

template <int LA, int LB, int LC, int LD, bool GEN, typename R>
__device__ __forceinline__ void row_body(const FockArgs& a)
{
    using C = EriClass<LA, LB, LC, LD>;
    using Store = RowStore<LA, LB, LC, LD, GEN>;
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1, NC = 2 * LC + 1, ND = 2 * LD + 1;
    constexpr int NROW = row_elements<LA, LB, LC, LD, GEN>;
    constexpr int DS = Store::d_registers ? 1 : kColumn;
    constexpr bool f32 = sizeof(R) == sizeof(float);
    // the straight-line code of a step of the large classes (up to hundreds of
    // KB) does not fit the instruction caches, least of all beside other
    // classes' kernels: the warps of a block walk their items in step, so that it
    // is fetched once for all of them ((H2O)27 / def2-TZVP build 236 -> 228 ms;
    // each class by itself 3% slower to 18% faster)
    constexpr bool LOCK = !Store::sums;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    extern __shared__ __align__(16) char shared[];
    R* sboys = reinterpret_cast<R*>(shared);
    double* sacc = reinterpret_cast<double*>(shared + (boys_stride<R> * (int)sizeof(R) + 15) / 16 * 16);
    double* acc = sacc + warp * (kColumn * NROW) + lane;
    double rdc[Store::d_registers ? NROW : 1];
    double* dc = Store::d_registers ? rdc : acc + kWarpsPerBlock * kColumn * NROW;
    stage_boys<LA + LB + LC + LD>(a, sboys);
#pragma unroll 1
    for (;;) {
        WorkItem w;
        int steps;
        if constexpr (LOCK) {
            // four consecutive items for the block's warps, walked in step
            __shared__ int first;
            __syncthreads();
            if (threadIdx.x == 0) first = atomicAdd(a.counter, kWarpsPerBlock);
            __syncthreads();
            const int base = first;
            if (base >= a.nitems) return;
            steps = 0;
            for (int v = 0; v < kWarpsPerBlock; v++) {
                const int it = min(base + v, a.nitems - 1);
                const WorkItem x = a.items[it];
                steps = max(steps, x.kend - x.bra);
                if (v == warp) {
                    w = x;
                    if (base + v >= a.nitems) w.kend = w.bra;  // no item for this warp
                }
            }
        } else {
            int it = 0;
            if (lane == 0) it = atomicAdd(a.counter, 1);
            it = __shfl_sync(0xffffffffu, it, 0);
            if (it >= a.nitems) return;
            w = a.items[it];
            steps = w.kend - w.bra;
        }
        const bool diag = (w.blocks & 0xffff) == ((unsigned)w.blocks >> 16);
        const PairBlockDev& bb = a.blocks[w.blocks & 0xffff];
        const PairBlockDev& kb = a.blocks[(unsigned)w.blocks >> 16];
        const MolDev m = a.mols ? a.mols[bb.mol] : a.mol;
        const int kl = w.kbeg + lane, jj = min(kl, kb.npairs - 1);
        int4 head = __ldg(bb.rhead + w.bra);
        QuartetAO o;
        o.nlp = m.nl[LA];
        o.nlq = m.nl[LB];
        o.nlr = m.nl[LC];
        o.nls = m.nl[LD];
        o.q0 = head.z;
        o.r0 = __ldg(kb.ao + jj);
        o.s0 = __ldg(kb.ao + kb.npairs + jj);
        const double s_ket = (o.r0 == o.s0) ? 0.5 : 1.0;
        const PairViewT<R> ket = make_view(kb, jj, __ldg(kb.nuse + jj), R());
        if constexpr (Store::sums) begin_row<NB, NC, ND, GEN, DS>(o, m, a.cj, a.ck, acc, dc);
        bool any = false;
#pragma unroll 1
        for (int x = 0; x < steps; x++) {
            if constexpr (LOCK) {
                __syncthreads();
                if (w.bra + x >= w.kend) continue;
            }
            const int q = w.bra + x;
            const int4 h = head;  // the next pair's header is read a step ahead
            if (q + 1 < w.kend) head = __ldg(bb.rhead + q + 1);
            const int bx = h.w & 15;
            // the kets this launch admits for the bra pair (see item_range)
            int k0 = diag ? h.x : 0, k1 = 0;
            if (a.ith >= bx) k1 = __ldg(kb.bin_off + min(a.ith - bx, 15) + 1);
            if (k1 <= w.kbeg) {  // ascending bins: nor any later pair's
                if (!LOCK) break;
                w.kend = q;
                continue;
            }
            if (a.ith32 >= 0) {
                const int kmid = (a.ith32 <= bx) ? 0 : __ldg(kb.bin_off + min(a.ith32 - bx, 16));
                if (f32)
                    k0 = max(k0, kmid);
                else
                    k1 = min(k1, kmid);
            }
            if (max(k0, w.kbeg) >= min(k1, w.kbeg + 32)) continue;
            const bool act = kl >= k0 && kl < k1;
            any = any || act;
            o.p0 = h.y;
            double s = act ? s_ket : 0.0;
            if (o.p0 == o.q0) s *= 0.5;
            if (diag && kl == h.x) s *= 0.5;
            if constexpr (Store::stream) {
                StreamSink<NA, NB, NC, ND, R> sink(o, m, a.cj, a.ck, s);
                eri_compute<C>(make_row_view(bb, q, h.w >> 4, R()), ket, sboys, a.omega2, sink);
                sink.finish(lane);
            } else {
                R g[C::NSPH];
                ArraySink<NA * NB, NC, ND, R> sink{g};
                eri_compute<C>(make_row_view(bb, q, h.w >> 4, R()), ket, sboys, a.omega2, sink);
                double f[C::NSPH];
#pragma unroll
                for (int t = 0; t < C::NSPH; t++) f[t] = (double)g[t];
                if constexpr (Store::sums)
                    digest_row<NA, NB, NC, ND, GEN, DS>(f, s, lane, o, m, a.cj, a.ck, acc, dc);
                else
                    digest<NA, NB, NC, ND, GEN ? MODE_FOCK_GEN : MODE_FOCK_SYM>(
                        f, s, lane, o.p0, o.nlp, o.q0, o.nlq, o.r0, o.nlr, o.s0, o.nls, m, a.cj, a.ck);
            }
        }
        if constexpr (Store::sums) {
            if (any) flush_row<NB, NC, ND, GEN>(o, m, a.cj, a.ck, acc);
        }
    }
}

// Kernel variants of a class: row items (plain builds) and pair items (extended
// builds), each for symmetric and general densities; the ERI tensor is with the
// general pair items.  Each is a kernel of its own, so that it has only its own
// live values.
enum KernelVariant { ROWS_SYM = 0, ROWS_GEN = 1, PAIRS_SYM = 2, PAIRS_GEN = 3 };
constexpr int kNumVariants = 4;

template <int LA, int LB, int LC, int LD, int V, typename R>
__device__ __forceinline__ void kernel_body(const FockArgs& a, const int mode)
{
    if constexpr (V >= PAIRS_SYM)
        quartet_body<LA, LB, LC, LD, V == PAIRS_GEN, R>(a, mode);
    else
        row_body<LA, LB, LC, LD, V == ROWS_GEN, R>(a);
}

template <int MB, int LA, int LB, int LC, int LD, int V, typename R>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, MB) quartet_kernel(const FockArgs a, const int mode)
{
    kernel_body<LA, LB, LC, LD, V, R>(a, mode);
}

// without a minimum of resident blocks (a minimum of 1 is not the same: it lets
// the compiler take far more registers)
template <int LA, int LB, int LC, int LD, int V, typename R>
__global__ void __launch_bounds__(32 * kWarpsPerBlock) quartet_kernel_free(const FockArgs a, const int mode)
{
    kernel_body<LA, LB, LC, LD, V, R>(a, mode);
}

// the kernel of a class, variant and precision, and its dynamic shared memory
template <int LA, int LB, int LC, int LD, int V, typename R>
constexpr auto quartet_kernel_of()
{
    constexpr int mb = BlocksHint<LA, LB, LC, LD, V>::value;
    if constexpr (mb > 0)
        return &quartet_kernel<(mb > 0 ? mb : 1), LA, LB, LC, LD, V, R>;
    else
        return &quartet_kernel_free<LA, LB, LC, LD, V, R>;
}

template <int LA, int LB, int LC, int LD, int V, typename R>
constexpr int quartet_shared_bytes()
{
    if constexpr (V >= PAIRS_SYM)
        return 0;
    else
        return row_shared_bytes<LA, LB, LC, LD, V == ROWS_GEN, R>();
}

template <int LA, int LB, int LC, int LD, int V, typename R>
void launch_quartet_as(int mode, const FockArgs& a, int grid, cudaStream_t st)
{
    quartet_kernel_of<LA, LB, LC, LD, V, R>()<<<grid, 32 * kWarpsPerBlock,
                                               quartet_shared_bytes<LA, LB, LC, LD, V, R>(), st>>>(a, mode);
}

template <int LA, int LB, int LC, int LD, int V>
void launch_quartet(int mode, const FockArgs& a, int grid, cudaStream_t st)
{
    if (mode & MODE_F32)
        launch_quartet_as<LA, LB, LC, LD, V, float>(mode, a, grid, st);
    else
        launch_quartet_as<LA, LB, LC, LD, V, double>(mode, a, grid, st);
}

// Resident blocks per SM (also sets the kernel's limit of dynamic shared
// memory on the current device: called before its first launch there).
template <int LA, int LB, int LC, int LD, int V, typename R>
int occupancy_quartet_as()
{
    constexpr int bytes = quartet_shared_bytes<LA, LB, LC, LD, V, R>();
    const auto kernel = quartet_kernel_of<LA, LB, LC, LD, V, R>();
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 32 * kWarpsPerBlock, bytes);
    return n;
}

template <int LA, int LB, int LC, int LD, int V>
int occupancy_quartet(bool f32)
{
    return f32 ? occupancy_quartet_as<LA, LB, LC, LD, V, float>() : occupancy_quartet_as<LA, LB, LC, LD, V, double>();
}

// max over all spherical components of (ab|ab) per pair (T4CScreener::partition)
template <int LA, int LB>
__global__ void __launch_bounds__(64) schwarz_kernel(const PairBlockDev* blocks, const int bid, const double* boys,
                                                     double* maxv)
{
    using C = EriClass<LA, LB, LA, LB>;
    const PairBlockDev b = blocks[bid];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.npairs) return;
    const PairView v = make_view(b, i);
    double f[C::NSPH];
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1;
    ArraySink<NA * NB, NA, NB, double> sink{f};
    C::compute(v, v, boys + (size_t)(2 * (LA + LB)) * BOYS_STRIDE, 0.0, sink);
    double mx = 0.0;
    for (int t = 0; t < C::NSPH; t++) mx = (f[t] > mx) ? f[t] : mx;
    maxv[i] = mx;
}

}  // namespace vlx
