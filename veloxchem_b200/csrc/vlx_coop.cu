// Warp-cooperative kernel for the quartet classes whose contracted buffer is
// too large for registers ((pd|pd), (dd|pp), (dd|sd), (dd|pd), (dd|dd) and the
// f classes).  One warp evaluates one shell quartet: the per-primitive
// recursion program generated by gen_coop.py (the same Obara-Saika steps as the
// compiled classes) runs level by level on a per-warp shared-memory array,
// lanes taking the independent operations of a level round-robin, and sums
// into the accumulators [e 0 | f 0]; the post-contraction steps are compiled
// per class (KetXform over the e rows, then BraXform over the ket components,
// lane-parallel); then the warp digests the spherical block into J/K (each
// lane owns some of the contracted outputs), or scatters it into the ERI
// tensor, or reduces its maximum (Schwarz).
#include "vlx_coop.cuh"

#include <algorithm>
#include <type_traits>

namespace vlx {

#include "xform.inc"

constexpr int coop_ncart(int l) { return (l + 1) * (l + 2) / 2; }
// e components [lb, la+lb] and f components [ld, lc+ld] of the accumulators
constexpr int coop_ne(int la, int lb)
{
    int n = 0;
    for (int l = lb; l <= la + lb; l++) n += coop_ncart(l);
    return n;
}

// geometry block appended to each warp's slot array
constexpr int kGeo = 24;  // 0-2 P-B, 3-5 Q-D, 6-8 W-P, 9-11 W-Q, 12 hiz, 13 hie, 14 rz, 15 rh,
                          // 16 hizh, 18-20 D-C, 21-23 B-A

// F_m(T) for one order from its Chebyshev table (no recursion: each lane of
// the warp evaluates one order of the same T); R = double, or float for the
// mixed-precision twin (float table, float arithmetic).
__device__ __forceinline__ double rsqrt_r(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_r(float x) { return rsqrtf(x); }
__device__ __forceinline__ double exp_r(double x) { return exp(x); }
__device__ __forceinline__ float exp_r(float x) { return expf(x); }

template <typename R>
__device__ __forceinline__ R boys_one(const int m, const R T, const R* __restrict__ tab)
{
    if (T < (R)BOYS_TMAX) {
        constexpr bool f32 = sizeof(R) == sizeof(float);
        constexpr int nc = f32 ? BOYS_NCOEF_F : BOYS_NCOEF, stride = f32 ? BOYS_STRIDE_F : BOYS_STRIDE;
        const int it = (int)(T * (R)BOYS_INV_H + (R)0.5);
        const R x = (R)(2 * BOYS_INV_H) * T - (R)(2 * it);
        const R* c = tab + m * stride + it * nc;
        R p = __ldg(c + nc - 1);
#pragma unroll
        for (int j = nc - 2; j >= 0; j--) p = p * x + __ldg(c + j);
        return p;
    }
    // F_0 = sqrt(pi / T) / 2 (erf(sqrt T) = 1 to working precision), then the
    // upward recursion, stable for T >= BOYS_TMAX > m + 1/2
    R f = (R)0.88622692545275801365 * rsqrt_r(T);
    const R h = (R)0.5 / T;
    const R et = exp_r(-T);
    for (int k = 0; k < m; k++) f = ((R)(2 * k + 1) * f - et) * h;
    return f;
}

// One level: lanes take the level's independent ops round-robin, four at a
// time with the records loaded before any operand (four independent chains).
template <typename R>
__device__ __forceinline__ R op_value(const int4 r, const R* __restrict__ S, const R* __restrict__ geo)
{
    const int kind = (r.w >> 2) & 0x3f, ax = r.w & 3;
    const int x = (r.x >> 16) & 0xffff, y = r.y & 0xffff;
    if (kind <= 1) {
        const int u = (r.y >> 16) & 0xffff, v = r.z & 0xffff, w = (r.z >> 16) & 0xffff;
        const int c1 = (r.w >> 8) & 0xff, c2 = (r.w >> 16) & 0xff;
        R val = geo[kind * 3 + ax] * S[x] + geo[6 + kind * 3 + ax] * S[y];
        if (c1) val += (R)c1 * geo[12 + kind] * (S[u] - geo[14 + kind] * S[v]);
        if (c2) val += (R)c2 * geo[16] * S[w];
        return val;
    }
    return S[r.x & 0xffff] + S[x];  // kind 2: accumulate
}

template <typename R>
__device__ __forceinline__ void run_ops(const int4* __restrict__ ops, R* __restrict__ S, const R* __restrict__ geo,
                                        const int first, const int last, const int lane)
{
    constexpr int U = 4;
    for (int base = first + lane; base < last; base += 32 * U) {
        int4 r[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int o = base + 32 * u;
            r[u] = (o < last) ? ops[o] : make_int4(0, 0, 0, -1);
        }
        R val[U];
#pragma unroll
        for (int u = 0; u < U; u++) val[u] = (r[u].w >= 0) ? op_value(r[u], S, geo) : (R)0;
#pragma unroll
        for (int u = 0; u < U; u++)
            if (r[u].w >= 0) S[r[u].x & 0xffff] = val[u];
    }
}

// Sums the primitive quartets of (bra | ket) into the accumulators
// S[1 + ie nfp + jf] = [e_ie 0 | f_jf 0].
template <typename R>
__device__ void coop_body(const CoopClassDev& c, const int4* __restrict__ ops, const PairView& bra,
                          const PairView& ket, const R* __restrict__ boys, const double om2, R* __restrict__ S,
                          R* __restrict__ geo, const int lane)
{
    const int L = c.la + c.lb + c.lc + c.ld;
    for (int t = lane; t <= c.nacc; t += 32) S[t] = (R)0;
    __syncwarp();
    const int kb = bra.nprim(), kk = ket.nprim();
    for (int pk = 0; pk < kk; pk++) {
        const double eta = ket.zeta(pk), hie = ket.hiz(pk), kcd = ket.kfac(pk);
        const double Qx = ket.px(pk), Qy = ket.py(pk), Qz = ket.pz(pk);
        for (int pb = 0; pb < kb; pb++) {
            const double zeta = bra.zeta(pb);
            const double PQx = bra.px(pb) - Qx, PQy = bra.py(pb) - Qy, PQz = bra.pz(pb) - Qz;
            const double r = rsqrt(zeta + eta);
            const double inv = r * r;
            const double rz = eta * inv, rh = zeta * inv;
            const double T = zeta * rz * (PQx * PQx + PQy * PQy + PQz * PQz);
            __syncwarp();  // previous iteration's reads of geo / F slots are done
            if (lane <= L) {
                const int fs = __ldg(c.fslots + lane);
                if (fs > 0) {
                    // erf-attenuated operator: s^(2m+1) F_m(s^2 T), s^2 = om2 / (om2 + rho)
                    double s2 = 1.0, sc = 1.0;
                    if (om2 > 0.0) {
                        s2 = om2 / (om2 + zeta * rz);
                        sc = sqrt(s2);
                        for (int k = 0; k < lane; k++) sc *= s2;
                    }
                    S[fs] = (R)(bra.kfac(pb) * kcd * r * sc) * boys_one<R>(lane, (R)(T * s2), boys);
                }
            }
            if (lane == 0) {
                geo[0] = (R)(bra.pbx(pb));
                geo[1] = (R)(bra.pby(pb));
                geo[2] = (R)(bra.pbz(pb));
                geo[3] = (R)(ket.pbx(pk));
                geo[4] = (R)(ket.pby(pk));
                geo[5] = (R)(ket.pbz(pk));
                geo[6] = (R)(-rz * PQx);
                geo[7] = (R)(-rz * PQy);
                geo[8] = (R)(-rz * PQz);
                geo[9] = (R)(rh * PQx);
                geo[10] = (R)(rh * PQy);
                geo[11] = (R)(rh * PQz);
                geo[12] = (R)(bra.hiz(pb));
                geo[13] = (R)(hie);
                geo[14] = (R)(rz);
                geo[15] = (R)(rh);
                geo[16] = (R)(0.5 * inv);
            }
            __syncwarp();
            for (int l = 1; l <= c.nblev; l++) {
                run_ops(ops, S, geo, __ldg(c.boff + l), __ldg(c.boff + l + 1), lane);
                __syncwarp();
            }
        }
    }
}

// Ket HRR + spherical transform of every e row (lane-parallel), then bra HRR
// + spherical transform of every ket component: fout[((i NB + j) NC + k) ND + l].
template <typename R, int LA, int LB, int LC, int LD>
__device__ __forceinline__ void coop_post(R* __restrict__ S, R* __restrict__ fout, const PairView& bra,
                                          const PairView& ket, const int lane)
{
    constexpr int NE = coop_ne(LA, LB), NF = coop_ne(LC, LD), NFP = NF | 1;
    constexpr int NSCD = (2 * LC + 1) * (2 * LD + 1), XS = NSCD | 1;
    const R* acc = S + 1;
    R* X = S + 1 + NE * NFP;
    const R DCx = (R)ket.abx(), DCy = (R)ket.aby(), DCz = (R)ket.abz();
    for (int ie = lane; ie < NE; ie += 32) KetXform<LC, LD>::run(acc + ie * NFP, X + ie * XS, 1, DCx, DCy, DCz);
    __syncwarp();
    const R BAx = (R)bra.abx(), BAy = (R)bra.aby(), BAz = (R)bra.abz();
    for (int kl = lane; kl < NSCD; kl += 32) BraXform<LA, LB>::run(X + kl, XS, fout + kl, NSCD, BAx, BAy, BAz);
    __syncwarp();
}

// Density sub-blocks of one quartet staged in shared memory: six (symmetric
// density) or twelve (general density) blocks, element (x, y) of block XY at
// XY[x * ny + y].
__host__ __device__ __forceinline__ int dstage_size(int NA, int NB, int NC, int ND)
{
    return 2 * (NA * NB + NC * ND + NB * ND + NB * NC + NA * ND + NA * NC);
}

// Cooperative J/K digestion: the density blocks are staged first (all lanes,
// independent loads), then the NA NB + NC ND + NA NC + NA ND + NB NC + NB ND
// contracted outputs are dealt over the lanes, reading f and D from shared
// memory, and each output is one atomic add (two for general densities).
template <typename R, int NA, int NB, int NC, int ND>
__device__ void coop_digest(const R* __restrict__ f, double* __restrict__ dst, const double s, const int lane,
                            const int p0, const int nlp, const int q0, const int nlq, const int r0, const int nlr,
                            const int s0, const int nls, const MolDev& m, const double cjw, const double ckw,
                            const int mode)
{
    const double* __restrict__ D = m.D;
    double* F = m.F;
    const size_t n = (size_t)m.nao;
    const bool gen = (mode == MODE_FOCK_GEN);
    // block descriptors: (row base, row stride, rows, col base, col stride, cols)
    const int desc[12][6] = {{p0, nlp, NA, q0, nlq, NB}, {r0, nlr, NC, s0, nls, ND}, {q0, nlq, NB, s0, nls, ND},
                             {q0, nlq, NB, r0, nlr, NC}, {p0, nlp, NA, s0, nls, ND}, {p0, nlp, NA, r0, nlr, NC},
                             {q0, nlq, NB, p0, nlp, NA}, {s0, nls, ND, r0, nlr, NC}, {s0, nls, ND, q0, nlq, NB},
                             {r0, nlr, NC, q0, nlq, NB}, {s0, nls, ND, p0, nlp, NA}, {r0, nlr, NC, p0, nlp, NA}};
    constexpr int off[13] = {0,
                             NA * NB,
                             NA * NB + NC * ND,
                             NA * NB + NC * ND + NB * ND,
                             NA * NB + NC * ND + NB * ND + NB * NC,
                             NA * NB + NC * ND + NB * ND + NB * NC + NA * ND,
                             NA * NB + NC * ND + NB * ND + NB * NC + NA * ND + NA * NC,
                             2 * NA * NB + NC * ND + NB * ND + NB * NC + NA * ND + NA * NC,
                             2 * NA * NB + 2 * NC * ND + NB * ND + NB * NC + NA * ND + NA * NC,
                             2 * NA * NB + 2 * NC * ND + 2 * NB * ND + NB * NC + NA * ND + NA * NC,
                             2 * NA * NB + 2 * NC * ND + 2 * NB * ND + 2 * NB * NC + NA * ND + NA * NC,
                             2 * NA * NB + 2 * NC * ND + 2 * NB * ND + 2 * NB * NC + 2 * NA * ND + NA * NC,
                             2 * (NA * NB + NC * ND + NB * ND + NB * NC + NA * ND + NA * NC)};
    const int nb = gen ? 12 : 6;
#pragma unroll
    for (int b = 0; b < 12; b++) {
        if (b >= nb) break;
        const int rb = desc[b][0], rs = desc[b][1], cb = desc[b][3], cs = desc[b][4], nc = desc[b][5];
        const int cnt = off[b + 1] - off[b];
        for (int e = lane; e < cnt; e += 32) {
            const int x = e / nc, y = e - x * nc;
            dst[off[b] + e] = __ldg(D + (size_t)(rb + x * rs) * n + cb + y * cs);
        }
    }
    __syncwarp();
    const double *Dpq = dst + off[0], *Drs = dst + off[1], *Dqs = dst + off[2], *Dqr = dst + off[3],
                 *Dps = dst + off[4], *Dpr = dst + off[5], *Dqp = dst + off[6], *Dsr = dst + off[7],
                 *Dsq = dst + off[8], *Drq = dst + off[9], *Dsp = dst + off[10], *Drp = dst + off[11];
    auto add = [&](int r, int cc, double v) { red_add(F + (size_t)r * n + cc, v); };
    auto fv = [&](int i, int j, int k, int l) { return (double)f[((i * NB + j) * NC + k) * ND + l]; };
    const int nJ1 = (cjw != 0.0) ? NA * NB : 0, nJ2 = (cjw != 0.0) ? NC * ND : 0;
    const int nK = (ckw != 0.0) ? NA * NC + NA * ND + NB * NC + NB * ND : 0;
    const int total = nJ1 + nJ2 + nK;
    const double cj = cjw * s, ck = ckw * s;
    for (int o = lane; o < total; o += 32) {
        if (o < nJ1) {
            const int i = o / NB, j = o % NB;
            double v = 0.0;
            for (int k = 0; k < NC; k++)
                for (int l = 0; l < ND; l++) {
                    double d = Drs[k * ND + l];
                    if (gen) d += Dsr[l * NC + k];
                    v = fma(fv(i, j, k, l), d, v);
                }
            add(p0 + i * nlp, q0 + j * nlq, cj * v);
            if (gen) add(q0 + j * nlq, p0 + i * nlp, cj * v);
            continue;
        }
        int q = o - nJ1;
        if (q < nJ2) {
            const int k = q / ND, l = q % ND;
            double v = 0.0;
            for (int i = 0; i < NA; i++)
                for (int j = 0; j < NB; j++) {
                    double d = Dpq[i * NB + j];
                    if (gen) d += Dqp[j * NA + i];
                    v = fma(fv(i, j, k, l), d, v);
                }
            add(r0 + k * nlr, s0 + l * nls, cj * v);
            if (gen) add(s0 + l * nls, r0 + k * nlr, cj * v);
            continue;
        }
        q -= nJ2;
        double v = 0.0, w = 0.0;
        if (q < NA * NC) {  // F_PR += f D_QS
            const int i = q / NC, k = q % NC;
            for (int j = 0; j < NB; j++)
                for (int l = 0; l < ND; l++) {
                    const double x = fv(i, j, k, l);
                    v = fma(x, Dqs[j * ND + l], v);
                    if (gen) w = fma(x, Dsq[l * NB + j], w);
                }
            add(p0 + i * nlp, r0 + k * nlr, ck * v);
            if (gen) add(r0 + k * nlr, p0 + i * nlp, ck * w);
            continue;
        }
        q -= NA * NC;
        if (q < NA * ND) {  // F_PS += f D_QR
            const int i = q / ND, l = q % ND;
            for (int j = 0; j < NB; j++)
                for (int k = 0; k < NC; k++) {
                    const double x = fv(i, j, k, l);
                    v = fma(x, Dqr[j * NC + k], v);
                    if (gen) w = fma(x, Drq[k * NB + j], w);
                }
            add(p0 + i * nlp, s0 + l * nls, ck * v);
            if (gen) add(s0 + l * nls, p0 + i * nlp, ck * w);
            continue;
        }
        q -= NA * ND;
        if (q < NB * NC) {  // F_QR += f D_PS
            const int j = q / NC, k = q % NC;
            for (int i = 0; i < NA; i++)
                for (int l = 0; l < ND; l++) {
                    const double x = fv(i, j, k, l);
                    v = fma(x, Dps[i * ND + l], v);
                    if (gen) w = fma(x, Dsp[l * NA + i], w);
                }
            add(q0 + j * nlq, r0 + k * nlr, ck * v);
            if (gen) add(r0 + k * nlr, q0 + j * nlq, ck * w);
            continue;
        }
        q -= NB * NC;
        {  // F_QS += f D_PR
            const int j = q / ND, l = q % ND;
            for (int i = 0; i < NA; i++)
                for (int k = 0; k < NC; k++) {
                    const double x = fv(i, j, k, l);
                    v = fma(x, Dpr[i * NC + k], v);
                    if (gen) w = fma(x, Drp[k * NA + i], w);
                }
            add(q0 + j * nlq, s0 + l * nls, ck * v);
            if (gen) add(s0 + l * nls, q0 + j * nlq, ck * w);
        }
    }
}

// Op records staged in shared memory (bytes) when the program is at most this long.
constexpr int kStageOpsMax = 32 * 1024;
__host__ __device__ __forceinline__ bool coop_stage_ops(int nbody) { return nbody * 16 <= kStageOpsMax; }

// Shared memory of one warp: S (nslots values), geo, the spherical block
// (R each), then the staged density blocks (double, 8-byte aligned).
__host__ __device__ __forceinline__ size_t coop_warp_bytes(int nslots, int nsph, int ndst, size_t rsize)
{
    // multiple of 16 bytes, so that the staged 16-byte op records after the warps' arrays are aligned
    return (((nslots + kGeo + nsph) * rsize + 7) / 8 * 8 + (size_t)ndst * sizeof(double) + 15) / 16 * 16;
}

template <typename R, int LA, int LB, int LC, int LD>
__global__ void coop_quartet_kernel(const FockArgs a, const CoopClassDev c, const int mode)
{
    extern __shared__ double smem[];
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1, NC = 2 * LC + 1, ND = 2 * LD + 1;
    constexpr int nsph = NA * NB * NC * ND;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t wb = coop_warp_bytes(c.nslots, nsph, dstage_size(NA, NB, NC, ND), sizeof(R));
    char* base = reinterpret_cast<char*>(smem) + (size_t)warp * wb;
    R* S = reinterpret_cast<R*>(base);
    R* geo = S + c.nslots;
    R* fout = geo + kGeo;
    double* dstage = reinterpret_cast<double*>(base + ((c.nslots + kGeo + nsph) * sizeof(R) + 7) / 8 * 8);
    const R* boys = std::is_same<R, float>::value ? reinterpret_cast<const R*>(a.boys_f)
                                                  : reinterpret_cast<const R*>(a.boys);
    const int dmode = mode & 3;
    // the per-primitive op records are re-read for every primitive quartet:
    // small programs are staged once per block behind the warps' arrays
    const int4* ops = c.ops;
    if (coop_stage_ops(c.nbody)) {
        int4* st = reinterpret_cast<int4*>(reinterpret_cast<char*>(smem) + (size_t)(blockDim.x >> 5) * wb);
        for (int o = threadIdx.x; o < c.nbody; o += blockDim.x) st[o] = __ldg(c.ops + o);
        __syncthreads();
        ops = st;
    }
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
        const int nlp = m.nl[LA], nlq = m.nl[LB], nlr = m.nl[LC], nls = m.nl[LD];
        const PairView bra = make_view(bb, w.bra);
        const int p0 = __ldg(bb.ao + w.bra), q0 = __ldg(bb.ao + bb.npairs + w.bra);
        constexpr bool F32 = std::is_same<R, float>::value;
        int k0, k1;
        // with density screening the precision is decided per quartet below
        item_range(a, bb, kb, w, F32 && !a.dsh, k0, k1);
        int P = 0, Q = 0;
        float qpq = 0.0f, dpq = 0.0f;
        if (a.dsh) {
            P = __ldg(bb.sh + w.bra);
            Q = __ldg(bb.sh + bb.npairs + w.bra);
            qpq = __ldg(bb.q + w.bra);
            dpq = __ldg(a.dsh + (size_t)P * a.nsh + Q);
            k1 = density_ket_end(a, P, Q, qpq, dpq, kb, F32, k1);
        }
        for (int j = k0; j < k1; j++) {
            // the same bound on every lane: the whole warp keeps or skips the quartet
            if (a.dsh && !quartet_kept(a, quartet_bound(a, P, Q, qpq, dpq, kb, j), F32)) continue;
            const PairView ket = make_view(kb, j);
            if (a.qstat && lane == 0) {
                atomicAdd(a.qstat, 1ull);
                atomicAdd(a.qstat + 1, (unsigned long long)(bra.kuse * ket.kuse));
            }
            coop_body<R>(c, ops, bra, ket, boys, a.omega2, S, geo, lane);
            coop_post<R, LA, LB, LC, LD>(S, fout, bra, ket, lane);
            const int r0 = __ldg(kb.ao + j), s0 = __ldg(kb.ao + kb.npairs + j);
            if (dmode == MODE_ERI) {
                const size_t n = (size_t)m.nao;
                double* e = a.eri;
                for (int t = lane; t < nsph; t += 32) {
                    const int i = t / (NB * NC * ND), jb = (t / (NC * ND)) % NB, k = (t / ND) % NC, l = t % ND;
                    const size_t p = p0 + i * nlp, q = q0 + jb * nlq, r = r0 + k * nlr, u = s0 + l * nls;
                    const double v = (double)fout[t];
                    e[((p * n + q) * n + r) * n + u] = v;
                    e[((q * n + p) * n + r) * n + u] = v;
                    e[((p * n + q) * n + u) * n + r] = v;
                    e[((q * n + p) * n + u) * n + r] = v;
                    e[((r * n + u) * n + p) * n + q] = v;
                    e[((u * n + r) * n + p) * n + q] = v;
                    e[((r * n + u) * n + q) * n + p] = v;
                    e[((u * n + r) * n + q) * n + p] = v;
                }
            } else {
                double s = (p0 == q0) ? 0.5 : 1.0;
                if (r0 == s0) s *= 0.5;
                if (bbi == kbi && j == w.bra) s *= 0.5;
                // one density, or each density of a multi-density build in turn
                const int nd = a.dens.n > 0 ? a.dens.n : 1;
                for (int d = 0; d < nd; d++) {
                    MolDev md = m;
                    double cj = a.cj, ck = a.ck;
                    if (a.dens.n > 0) {
                        md.D = a.dens.D[d];
                        md.F = a.dens.F[d];
                        cj = a.dens.cj[d];
                        ck = a.dens.ck[d];
                    }
                    coop_digest<R, NA, NB, NC, ND>(fout, dstage, s, lane, p0, nlp, q0, nlq, r0, nlr, s0, nls, md, cj,
                                                   ck, dmode);
                    __syncwarp();  // the staged density blocks are reused by the next density
                }
            }
            __syncwarp();
        }
    }
}

template <int LA, int LB, int LC, int LD>
__global__ void coop_schwarz_kernel(const PairBlockDev* blocks, const int bid, const CoopClassDev c,
                                    const double* boys, double* maxv)
{
    extern __shared__ double smem[];
    constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1, NC = 2 * LC + 1, ND = 2 * LD + 1;
    constexpr int nsph = NA * NB * NC * ND;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t wb = coop_warp_bytes(c.nslots, nsph, dstage_size(NA, NB, NC, ND), sizeof(double));
    double* S = reinterpret_cast<double*>(reinterpret_cast<char*>(smem) + (size_t)warp * wb);
    double* geo = S + c.nslots;
    double* fout = geo + kGeo;
    const PairBlockDev b = blocks[bid];
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    for (int i = blockIdx.x * (blockDim.x >> 5) + warp; i < b.npairs; i += nwarps) {
        const PairView v = make_view(b, i);
        coop_body<double>(c, c.ops, v, v, boys, 0.0, S, geo, lane);
        coop_post<double, LA, LB, LC, LD>(S, fout, v, v, lane);
        double mx = 0.0;
        for (int t = lane; t < nsph; t += 32) mx = (fout[t] > mx) ? fout[t] : mx;
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) maxv[i] = mx;
        __syncwarp();
    }
}

namespace {

template <typename R, int LA, int LB, int LC, int LD>
void launch_q(int mode, const FockArgs& a, const CoopClassDev& c, int grid, int warps, size_t smem, cudaStream_t st)
{
    coop_quartet_kernel<R, LA, LB, LC, LD><<<grid, 32 * warps, smem, st>>>(a, c, mode);
}

template <int LA, int LB, int LC, int LD>
void launch_s(const PairBlockDev* blocks, int bid, const CoopClassDev& c, const double* boys, double* maxv, int grid,
              int warps, size_t smem, cudaStream_t st)
{
    coop_schwarz_kernel<LA, LB, LC, LD><<<grid, 32 * warps, smem, st>>>(blocks, bid, c, boys, maxv);
}

using QuartetLaunch = void (*)(int, const FockArgs&, const CoopClassDev&, int, int, size_t, cudaStream_t);

struct CoopEntry {
    int la, lb, lc, ld;
    QuartetLaunch quartet[2];  // FP64, FP32
    void (*schwarz)(const PairBlockDev*, int, const CoopClassDev&, const double*, double*, int, int, size_t,
                    cudaStream_t);
    const void* qfn[2];
    const void* sfn;
};

#define VLX_COOP_CLASS(A, B, C, D)                                                                     \
    {A, B, C, D, {&launch_q<double, A, B, C, D>, &launch_q<float, A, B, C, D>}, &launch_s<A, B, C, D>,  \
     {reinterpret_cast<const void*>(&coop_quartet_kernel<double, A, B, C, D>),                         \
      reinterpret_cast<const void*>(&coop_quartet_kernel<float, A, B, C, D>)},                         \
     reinterpret_cast<const void*>(&coop_schwarz_kernel<A, B, C, D>)},
const CoopEntry kCoopClasses[] = {
#include "coop_classes.inc"
};
#undef VLX_COOP_CLASS

const CoopEntry* coop_entry(const CoopClassDev& c)
{
    for (const CoopEntry& e : kCoopClasses)
        if (e.la == c.la && e.lb == c.lb && e.lc == c.lc && e.ld == c.ld) return &e;
    return nullptr;
}

}  // namespace

size_t coop_smem_per_warp(const CoopClassDev& c, bool f32)
{
    const int NA = 2 * c.la + 1, NB = 2 * c.lb + 1, NC = 2 * c.lc + 1, ND = 2 * c.ld + 1;
    return coop_warp_bytes(c.nslots, NA * NB * NC * ND, dstage_size(NA, NB, NC, ND),
                           f32 ? sizeof(float) : sizeof(double));
}

static size_t coop_block_bytes(const CoopClassDev& c, bool f32, int warps)
{
    return coop_smem_per_warp(c, f32) * warps + (coop_stage_ops(c.nbody) ? (size_t)c.nbody * 16 : 0);
}

int coop_warps_per_block(const CoopClassDev& c, bool f32)
{
    const size_t per = coop_smem_per_warp(c, f32);
    const size_t stage = coop_stage_ops(c.nbody) ? (size_t)c.nbody * 16 : 0;
    int w = 4;
    while (w > 1 && per * w + stage > 200 * 1024) w--;
    return w;
}

cudaError_t coop_prepare()
{
    for (const CoopEntry& e : kCoopClasses) {
        for (int f = 0; f < 2; f++) {
            cudaError_t r = cudaFuncSetAttribute(e.qfn[f], cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (r != cudaSuccess) return r;
        }
        cudaError_t r = cudaFuncSetAttribute(e.sfn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (r != cudaSuccess) return r;
    }
    return cudaSuccess;
}

int coop_blocks_per_sm(const CoopClassDev& c, bool f32)
{
    const CoopEntry* e = coop_entry(c);
    if (!e) return 1;
    int n = 0;
    const int w = coop_warps_per_block(c, f32);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, e->qfn[f32 ? 1 : 0], 32 * w, coop_block_bytes(c, f32, w));
    return n > 0 ? n : 1;
}

cudaError_t launch_coop_quartet(int mode, const FockArgs& a, const CoopClassDev& c, int grid, cudaStream_t st)
{
    const CoopEntry* e = coop_entry(c);
    if (!e) return cudaErrorInvalidValue;  // class without a compiled cooperative kernel
    const bool f32 = (mode & MODE_F32) != 0;
    const int w = coop_warps_per_block(c, f32);
    e->quartet[f32 ? 1 : 0](mode, a, c, grid, w, coop_block_bytes(c, f32, w), st);
    return cudaGetLastError();
}

cudaError_t launch_coop_schwarz(const PairBlockDev* blocks, int bid, int npairs, const CoopClassDev& c,
                                const double* boys, double* maxv, int nsm, cudaStream_t st)
{
    const CoopEntry* e = coop_entry(c);
    if (!e) return cudaErrorInvalidValue;
    const int w = coop_warps_per_block(c, false);
    const int grid = std::max(1, std::min((npairs + w - 1) / w, nsm * 4));
    e->schwarz(blocks, bid, c, boys, maxv, grid, w, coop_smem_per_warp(c, false) * w, st);
    return cudaGetLastError();
}

}  // namespace vlx
