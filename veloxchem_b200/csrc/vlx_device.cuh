// Device-side building blocks of the B200 four-centre Fock build:
//   * shell-pair views (ket: one pair per lane; bra: warp-uniform, from the
//     ket's layout, staged in shared memory, or in row order),
//   * the FP64 and FP32 Boys functions from Chebyshev tables,
//   * the ket range of a pair item and the per-quartet density test.
// The digestion and the work-queue kernels are in vlx_kernels.cuh, the per-class
// recursions (EriClass<la,lb,lc,ld>) are generated by gen_eri.py.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vlx_types.h"

namespace vlx {

// ---------------------------------------------------------------- pair views
// One primitive pair's fields, as the recursions read them.
template <typename R>
struct PrimRec {
    R zeta, hiz, kfac, px, py, pz, pbx, pby, pbz;
};

// Field order inside a pair block's primitive array, tiles of 32 pairs
// [tile][prim][field][pair of the tile] (primitive pairs of each shell pair
// sorted by |kfac| descending, the first nuse[pair] of them significant):
//   0 zeta = a + b            1 hiz = 1 / (2 zeta)
//   2 kfac = Na Nb S_ab sqrt(zeta) sqrt(2 / sqrt(pi))
//   3..5  P = (a A + b B) / zeta       6..8  P - B
// and per tile ab[3][pair of the tile] = B - A; ao[2][pair] = AO index of m = 0
// of A, B.  The FP32 view (mixed precision) reads the rounded copies, so its
// primitive loops load half the bytes and convert nothing.
template <typename R>
struct PairViewT {
    const R* __restrict__ prim;  // the pair's column of its tile
    const R* __restrict__ ab;
    int kuse;
    __device__ __forceinline__ R fld(int f, int p) const { return __ldg(prim + p * 288 + f * 32); }
    __device__ __forceinline__ int nprim() const { return kuse; }
    __device__ __forceinline__ R zeta(int p) const { return fld(0, p); }
    __device__ __forceinline__ R hiz(int p) const { return fld(1, p); }
    __device__ __forceinline__ R kfac(int p) const { return fld(2, p); }
    __device__ __forceinline__ R px(int p) const { return fld(3, p); }
    __device__ __forceinline__ R py(int p) const { return fld(4, p); }
    __device__ __forceinline__ R pz(int p) const { return fld(5, p); }
    __device__ __forceinline__ R pbx(int p) const { return fld(6, p); }
    __device__ __forceinline__ R pby(int p) const { return fld(7, p); }
    __device__ __forceinline__ R pbz(int p) const { return fld(8, p); }
    __device__ __forceinline__ PrimRec<R> rec(int p) const
    {
        return {zeta(p), hiz(p), kfac(p), px(p), py(p), pz(p), pbx(p), pby(p), pbz(p)};
    }
    __device__ __forceinline__ R abx() const { return __ldg(ab); }
    __device__ __forceinline__ R aby() const { return __ldg(ab + 32); }
    __device__ __forceinline__ R abz() const { return __ldg(ab + 64); }
};
using PairView = PairViewT<double>;
using PairViewF = PairViewT<float>;

// Offset of primitive 0, field 0 of pair i, and of its B - A.
__host__ __device__ __forceinline__ size_t prim_offset(int kprim, int i) { return (size_t)(i >> 5) * kprim * 288 + (i & 31); }
__host__ __device__ __forceinline__ size_t ab_offset(int i) { return (size_t)(i >> 5) * 96 + (i & 31); }

// The bra pair's primitive fields staged in shared memory for a work item
// (record of 10 per primitive: the 9 fields of PairView, padded to 16 bytes),
// so that the warp-uniform reads of the inner primitive loop are shared-memory
// broadcasts; B - A stays in global memory (read once per quartet).
template <typename R>
struct PairViewS {
    const R* s;
    const R* ab;  // the pair's column of its tile's B - A
    int kuse;
    __device__ __forceinline__ int nprim() const { return kuse; }
    __device__ __forceinline__ R zeta(int p) const { return s[p * 10 + 0]; }
    __device__ __forceinline__ R hiz(int p) const { return s[p * 10 + 1]; }
    __device__ __forceinline__ R kfac(int p) const { return s[p * 10 + 2]; }
    __device__ __forceinline__ R px(int p) const { return s[p * 10 + 3]; }
    __device__ __forceinline__ R py(int p) const { return s[p * 10 + 4]; }
    __device__ __forceinline__ R pz(int p) const { return s[p * 10 + 5]; }
    __device__ __forceinline__ R pbx(int p) const { return s[p * 10 + 6]; }
    __device__ __forceinline__ R pby(int p) const { return s[p * 10 + 7]; }
    __device__ __forceinline__ R pbz(int p) const { return s[p * 10 + 8]; }
    __device__ __forceinline__ PrimRec<R> rec(int p) const
    {
        return {zeta(p), hiz(p), kfac(p), px(p), py(p), pz(p), pbx(p), pby(p), pbz(p)};
    }
    __device__ __forceinline__ R abx() const { return __ldg(ab); }
    __device__ __forceinline__ R aby() const { return __ldg(ab + 32); }
    __device__ __forceinline__ R abz() const { return __ldg(ab + 64); }
};

// A bra pair of a row item: its records in row order (PairBlockDev::rprim),
// read as warp-uniform vector loads (5 instead of 9, of contiguous bytes).
template <typename R>
struct Vec2;
template <>
struct Vec2<double> {
    using type = double2;
};
template <>
struct Vec2<float> {
    using type = float2;
};
template <typename R>
struct PairViewR {
    using Vec = typename Vec2<R>::type;
    const R* __restrict__ s;   // the pair's first record of 10 values
    const R* __restrict__ ab;  // its B - A
    int kuse;
    __device__ __forceinline__ int nprim() const { return kuse; }
    __device__ __forceinline__ PrimRec<R> rec(int p) const
    {
        const Vec* v = reinterpret_cast<const Vec*>(s + p * 10);
        const Vec a = __ldg(v), b = __ldg(v + 1), c = __ldg(v + 2), d = __ldg(v + 3), e = __ldg(v + 4);
        return {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y, e.x};
    }
    __device__ __forceinline__ R abx() const { return __ldg(ab); }
    __device__ __forceinline__ R aby() const { return __ldg(ab + 1); }
    __device__ __forceinline__ R abz() const { return __ldg(ab + 2); }
};

// Bra primitive pairs a staged record holds at most (36: a pair of two
// six-primitive shells); pairs with more use the global-memory view.
constexpr int kStageBraMax = 36;

// Stages the kuse significant primitive records of the pair at `v` (all lanes
// of the warp take part; the caller synchronises the warp before reading).
template <typename R>
__device__ __forceinline__ void stage_bra(R* __restrict__ s, const PairViewT<R>& v, const int lane)
{
    for (int x = lane; x < v.kuse * 9; x += 32) {
        const int p = x / 9, f = x - p * 9;
        s[p * 10 + f] = v.fld(f, p);
    }
}

__device__ __forceinline__ PairView make_view(const PairBlockDev& b, int i)
{
    PairView v;
    v.prim = b.prim + prim_offset(b.kprim, i);
    v.ab = b.ab + ab_offset(i);
    v.kuse = __ldg(b.nuse + i);
    return v;
}

// Fock accumulation: a reduction without a returned value (red.global.add),
// which the L1TEX unit forwards to L2 without a write-back to the registers.
__device__ __forceinline__ void red_add(double* p, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "d"(v));
}
__device__ __forceinline__ void red_add(float* p, float v)
{
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "f"(v));
}

// ---------------------------------------------------------------- elementary functions
// 1 / sqrt(x) for positive normal x: the PTX approximation (about 20 bits) and
// one third-order Householder step, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - x y^2.
// The arguments here (exponent sums, Boys arguments) are never zero, negative
// or special, so the checks of the library function are not needed; relative
// error below 3e-16.
__device__ __forceinline__ double rsqrt_pos(const double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}

// ---------------------------------------------------------------- Boys function
// F_m(T) = int_0^1 t^{2m} exp(-T t^2) dt.  For T < BOYS_TMAX the highest order
// needed is a degree-9 polynomial in the local variable x in [-1, 1] of the
// interval around the table point nearest to T (Chebyshev fit generated on the
// host from the convergent series in long double, stored in the monomial basis
// of x, so one Horner chain of 9 FMAs evaluates it), and the lower orders follow
// by the stable downward recursion F_m = (2 T F_{m+1} + e^{-T}) / (2m + 1), with
// e^{-T} = e^{-T_k} e^{-x/4} from the table and a polynomial of degree 10 (its
// Chebyshev expansion; 6e-18), a third of the instructions of the library's
// exponential.  For T >= BOYS_TMAX, F_0 = sqrt(pi / T) / 2 (erf(sqrt T) = 1 to
// double precision) and the upward recursion F_{m+1} = ((2m + 1) F_m - e^{-T}) /
// (2T) is stable; e^{-T} is below 3e-17 of F_0 and F_1 there.
// The nearest integer of 2 T comes from adding 1.5 2^52, whose sum holds it in
// the low word: no conversion instructions.
// tabM: the BOYS_STRIDE values of order M (global or shared memory: the class
// kernels stage their order in shared memory).
// Against intervals by truncation, the library's exponential and reciprocal
// root, and a division beyond BOYS_TMAX: the (H2O)32 / def2-SVP build 43.0 -> 37.5
// ms (sum of its classes).
// F[m] = sc F_m(T), m = 0..M: the scale enters the highest order (or F_0) and
// e^{-T} once, and the recursions carry it to the other orders.
__device__ __forceinline__ double boys_exp(const double x, const int k, const double* __restrict__ tabM)
{
    double p = 2.6318062436936905e-13;
    p = fma(p, x, -1.0528720142264342e-11);
    p = fma(p, x, 3.7844176871668523e-10);
    p = fma(p, x, -1.2110133608598948e-08);
    p = fma(p, x, 3.390842016068632e-07);
    p = fma(p, x, -8.138020840527125e-06);
    p = fma(p, x, 0.00016276041666661556);
    p = fma(p, x, -0.002604166666665382);
    p = fma(p, x, 0.03125000000000001);
    p = fma(p, x, -0.25000000000000006);
    p = fma(p, x, 1.0);
    return p * tabM[BOYS_NINT * BOYS_NCOEF + k];
}

template <int M>
__device__ __forceinline__ void boys_scaled(const double T, const double sc, double* F,
                                            const double* __restrict__ tabM)
{
    static_assert(BOYS_INV_H == 2, "the local variable and boys_exp assume half-unit intervals");
    if (T < (double)BOYS_TMAX) {
        const double near = fma(T, (double)BOYS_INV_H, 6755399441055744.0);
        const int k = __double2loint(near);
        const double x = fma(T, 4.0, -2.0 * (near - 6755399441055744.0));
        const double2* c2 = reinterpret_cast<const double2*>(tabM + k * BOYS_NCOEF);
        double c[BOYS_NCOEF];
#pragma unroll
        for (int j = 0; j < BOYS_NCOEF / 2; j++) {
            const double2 v = c2[j];
            c[2 * j] = v.x;
            c[2 * j + 1] = v.y;
        }
        double p = c[BOYS_NCOEF - 1];
#pragma unroll
        for (int j = BOYS_NCOEF - 2; j >= 0; j--) p = fma(p, x, c[j]);
        F[M] = sc * p;
        if (M > 0) {
            const double t2 = 2.0 * T, et = sc * boys_exp(x, k, tabM);
#pragma unroll
            for (int m = M - 1; m >= 0; m--) F[m] = fma(t2, F[m + 1], et) * (1.0 / (2 * m + 1));
        }
    } else {
        const double r = rsqrt_pos(T);
        F[0] = (sc * 0.88622692545275801365) * r;
        if (M > 0) {
            // 1 / (2T) from the same root, with one correction step
            const double r2 = r * r, h = 0.5 * fma(r2, fma(-T, r2, 1.0), r2);
            const double et = (M > 1) ? sc * exp(-T) : 0.0;
#pragma unroll
            for (int m = 0; m < M; m++) F[m + 1] = fma((double)(2 * m + 1), F[m], -et) * h;
        }
    }
}

template <int M>
__device__ __forceinline__ void boys_function_tab(const double T, double* F, const double* __restrict__ tabM)
{
    boys_scaled<M>(T, 1.0, F, tabM);
}

// tab: the whole table (orders 0..BOYS_MMAX)
template <int M>
__device__ __forceinline__ void boys_function(const double T, double* F, const double* __restrict__ tab)
{
    boys_function_tab<M>(T, F, tab + (size_t)M * BOYS_STRIDE);
}

// FP32 Boys function for the mixed-precision path: the same scheme in float
// (polynomials of degree 7, and 5 for e^{-x/4}).  e^{-T} beyond BOYS_TMAX is below
// 3e-8 of F_m up to order 10.  1 / (2T) takes the correction step of the FP64
// branch: the root is good to 2 ulp only and enters every step of the upward
// recursion.  Largest relative error, measured up to T = 500 and bounded by
// (7 + 3 m) 6e-8: 2e-7 at order 1, 8e-7 at order 12 below BOYS_TMAX, 1.1e-6 beyond
// (without the step 3.2e-6).
template <int M>
__device__ __forceinline__ void boys_scaled_f(const float T, const float sc, float* F, const float* __restrict__ tabM)
{
    if (T < (float)BOYS_TMAX) {
        const float near = fmaf(T, (float)BOYS_INV_H, 12582912.0f);
        const int k = __float_as_int(near) - 0x4b400000;
        const float x = fmaf(T, 4.0f, -2.0f * (near - 12582912.0f));
        const float4* c4 = reinterpret_cast<const float4*>(tabM + k * BOYS_NCOEF_F);
        const float4 lo = c4[0], hi = c4[1];
        float p = hi.w;
        p = fmaf(p, x, hi.z);
        p = fmaf(p, x, hi.y);
        p = fmaf(p, x, hi.x);
        p = fmaf(p, x, lo.w);
        p = fmaf(p, x, lo.z);
        p = fmaf(p, x, lo.y);
        p = fmaf(p, x, lo.x);
        F[M] = sc * p;
        if (M > 0) {
            float q = -8.15923726e-06f;
            q = fmaf(q, x, 0.000163269706f);
            q = fmaf(q, x, -0.00260415605f);
            q = fmaf(q, x, 0.0312498089f);
            q = fmaf(q, x, -0.250000001f);
            q = fmaf(q, x, 1.00000001f);
            const float t2 = 2.0f * T, et = sc * q * tabM[BOYS_NINT * BOYS_NCOEF_F + k];
#pragma unroll
            for (int m = M - 1; m >= 0; m--) F[m] = fmaf(t2, F[m + 1], et) * (1.0f / (2 * m + 1));
        }
    } else {
        const float r = rsqrtf(T);
        F[0] = (sc * 0.886226925f) * r;
        if (M > 0) {
            const float r2 = r * r, h = 0.5f * fmaf(r2, fmaf(-T, r2, 1.0f), r2);
            const float et = (M > 10) ? sc * expf(-T) : 0.0f;
#pragma unroll
            for (int m = 0; m < M; m++) F[m + 1] = fmaf((float)(2 * m + 1), F[m], -et) * h;
        }
    }
}

// Kets of a work item admitted at run time: the kets of a pair block are
// sorted by Schwarz bin, so those with bin_bra + bin_ket <= ith are a prefix,
// and the FP32 ones (bin sum >= ith32) the tail of that prefix.  f32 selects
// the FP32 part [k0, k1), otherwise the FP64 part.
__device__ __forceinline__ void item_range(const FockArgs& a, const PairBlockDev& bb, const PairBlockDev& kb,
                                           const WorkItem& w, const bool f32, int& k0, int& k1)
{
    const int bx = __ldg(bb.bin + w.bra);
    const int kmax = a.ith - bx;
    const int kend = (kmax < 0) ? w.kbeg : min(w.kend, __ldg(kb.bin_off + min(kmax, 15) + 1));
    int kmid = kend;
    if (a.ith32 >= 0) {
        const int b32 = a.ith32 - bx;
        const int kb32 = (b32 <= 0) ? 0 : __ldg(kb.bin_off + min(b32, 16));
        kmid = max(w.kbeg, min(kend, kb32));
    }
    k0 = f32 ? kmid : w.kbeg;
    k1 = f32 ? kend : kmid;
}

// Density-weighted bound of the quartet (PQ|RS) for per-quartet screening
// (FockArgs::dsh): q_PQ q_RS max(|cj| max(d_PQ, d_RS), |ck| max(d_PR, d_PS,
// d_QR, d_QS)), the largest change any one integral of the quartet can make
// to an element of F.  P, Q, qpq and dpq = d_PQ belong to the bra pair.
__device__ __forceinline__ float quartet_bound(const FockArgs& a, const int P, const int Q, const float qpq,
                                               const float dpq, const PairBlockDev& kb, const int j)
{
    const int R = __ldg(kb.sh + j), S = __ldg(kb.sh + kb.npairs + j);
    const float* __restrict__ d = a.dsh;
    const size_t n = (size_t)a.nsh;
    const float drs = __ldg(d + R * n + S);
    const float dk = fmaxf(fmaxf(__ldg(d + P * n + R), __ldg(d + P * n + S)),
                           fmaxf(__ldg(d + Q * n + R), __ldg(d + Q * n + S)));
    const float cj = fabsf((float)a.cj), ck = fabsf((float)a.ck);
    return qpq * __ldg(kb.q + j) * fmaxf(cj * fmaxf(dpq, drs), ck * dk);
}

// End of the kets of a work item [.., k1) that can pass the density test of
// the launch of precision f32.  The kets of a pair block are sorted by
// Schwarz bin and a ket of bin b >= 1 has q_RS < 10^(1-b); every quartet bound
// of the item is at most cap q_RS with cap = q_PQ max(|cj| max(d_PQ, max d),
// |ck| max(rowmax_P, rowmax_Q)), so the kets from the first bin whose
// cap 10^(1-b) is below the launch's cutoff on all fail the per-quartet test
// and are not walked.  The factors 1.001 and 1.0001 cover the float rounding
// of the per-quartet bound and of the rounded-up Schwarz factors.
__device__ __forceinline__ int density_ket_end(const FockArgs& a, const int P, const int Q, const float qpq,
                                               const float dpq, const PairBlockDev& kb, const bool f32, const int k1)
{
    const float tau = f32 ? a.tau_skip : fmaxf(a.tau_skip, a.tau32);
    if (!(tau > 0.0f)) return k1;
    const float* __restrict__ row = a.dsh_row;
    const float cj = fabsf((float)a.cj), ck = fabsf((float)a.ck);
    const float cap = 1.001f * qpq *
                      fmaxf(cj * fmaxf(dpq, __ldg(row + a.nsh)), ck * fmaxf(__ldg(row + P), __ldg(row + Q)));
    float qb = 1.0001f;  // bound of q_RS in bin 1, then bins 2, 3, ...
    for (int b = 1; b <= 15; b++, qb *= 0.1f)
        if (cap * qb < tau) return min(k1, __ldg(kb.bin_off + b));
    return k1;
}

// Whether the launch of precision f32 evaluates a quartet of bound b.
__device__ __forceinline__ bool quartet_kept(const FockArgs& a, const float b, const bool f32)
{
    return b >= a.tau_skip && ((b < a.tau32) == f32);
}

template <int LA, int LB, int LC, int LD>
struct EriClass;

}  // namespace vlx
