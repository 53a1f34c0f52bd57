// fpsg_pair.cuh — the resident kernel for a Delta with an offset pattern.
//
// k_resident loads Delta's column entries for every element it computes.  When every
// nonzero Delta_kj lies at one of a few offsets |k - j| and all have one value (Pattern:
// uniform hopping on a lattice numbered row by row), the terms of element (i, j) are its
// neighbours in the matrix itself,
//     sum_k X_ik Delta_kj = w sum_q X(i, j +- off_q),
//     sum_k Delta_ik X_kj = w sum_q X(i +- off_q, j),
// at fixed distances from the element's own address: one shared load and one complex
// multiply-add under a mask bit each, contiguous in the row index, with no entries to
// load and no address arithmetic.  A thread's slot holds two elements, (i, j) and
// (i, j + 1), of neighbouring columns: with 1 among the offsets each is a neighbour of
// the other, and both share the row's mask, the diagonal term of row i and the address.
//
// Shared-memory wavefronts per 64 elements and stage (FP32, two offsets), against
// k_resident's columns at P = 2:    neighbours 28 (36 with the own element), column
// entries 0 (24), state 4 (4), diagonal terms 2 (4), stores 8 (8): 42 against 78.
// FP32 arithmetic runs on the two-wide instructions, a complex number per instruction.
// 10x10 grid, FP32, 16384 trajectories x 41 steps: 189.0 -> 113.5 ms
// The FP64 instances spill at 128 registers, the fullest, <256, 5, split>, 600 bytes of stores and
// 388 of loads per thread; the FP32 ones that forward runs take do not.
//
// Otherwise the kernel is k_resident: M stacked spin matrices per CTA (one spin per CTA
// of a 2-CTA cluster in split mode), X double-buffered in shared memory, the state at the
// start of the step by slot, the partner's next Delta_jj written by the owner of each
// diagonal element.
#pragma once
#include <vector>
#include "fpsg_kernels.cuh"

namespace fpsg {

// A slot: i | j << 10 | m << 20 (element (i, j), i <= j, of matrix m) and its flags: the
// masks of columns j, j + 1 and row i (2 NS bits each) and PAIR_ONE when the slot holds
// (i, j) alone.
constexpr uint32_t PAIR_ONE = 1u << 30;
constexpr uint32_t PAIR_NONE = 1u << 31;             // an empty slot
constexpr int PAIR_NMAX = 1023;                      // sites
constexpr int PAIR_MMAX = 4095;                      // matrices per CTA

// Host order of a matrix's slots (i | j << 16, bit 31: alone; ~0: empty).  A warp takes 32
// consecutive slots and reads without bank conflicts when they are consecutive rows of one
// column pair.  Slots with diagonal elements come first, so that the partner spin's next
// diagonal is on its way early in the pass: the diagonal elements of odd columns, which no
// pair covers, and a trailing partial 32 x 32 block (filled up to whole warps); then each
// full diagonal block as 8 warps of two column pairs, (2p, 2p + 1) with rows 0 .. 2p and
// (30 - 2p, 31 - 2p) with rows 0 .. 30 - 2p, 32 slots in all; then the 32-row segments of
// the columns right of their block.
inline std::vector<uint32_t> pair_slot_order(int n)
{
    std::vector<uint32_t> o;
    auto put = [&](int i, int j, bool one) { o.push_back((uint32_t)i | ((uint32_t)j << 16) | (one ? PAIR_NONE : 0u)); };
    for (int j = 1; j < n; j += 2) put(j, j, true);
    const int r1 = n / 32 * 32;
    for (int j = r1; j < n; j += 2)
        for (int i = r1; i <= j; ++i) put(i, j, j + 1 >= n);
    while (r1 > 0 && o.size() % 32) o.push_back(~0u);
    for (int r = 0; r < r1; r += 32)
        for (int p = 0; p < 8; ++p) {
            for (int i = r; i <= r + 2 * p; ++i) put(i, r + 2 * p, false);
            for (int i = r; i <= r + 30 - 2 * p; ++i) put(i, r + 30 - 2 * p, false);
        }
    for (int r = 0; r < r1; r += 32)
        for (int j = r + 32; j < n; j += 2)
            for (int i = r; i < r + 32; ++i) put(i, j, j + 1 >= n);
    return o;
}

template <typename R>
__host__ __device__ __forceinline__ ResLayout<R> pair_layout(int n, int M, int slots, bool comp, int max_off,
                                                             bool dense_coul, bool coul_smem, bool split)
{
    ResLayout<R> L;
    const size_t RP = (size_t)((M * n) | 1);
    // masked neighbours may lie up to max_off + 1 columns outside X; what is read there
    // is discarded, but it must stay inside the allocation
    const size_t guard = sizeof(cplx<R>) * RP * (size_t)(max_off + 1);
    size_t o = 0;
    L.rho = o;  o = align16(o + sizeof(cplx<R>) * 2 * (size_t)slots);
    if (o < guard) o = align16(guard);
    L.x = o;    o = align16(o + sizeof(cplx<R>) * 2 * (size_t)n * RP);
    const size_t x_end = o;
    L.dd = o;   o = align16(o + sizeof(R) * 6 * ((size_t)M * n + 1));     // Delta_jj and the other spin's diagonal, x3
    L.dg = o;   o = align16(o + sizeof(R) * 2 * ((size_t)M * n + 1));     // the diagonal, double-buffered
    L.sd = o;   o = align16(o + sizeof(R) * 4 * (size_t)n + 32);          // tM_jj, U_jj, extPot_jj, pulse; 3 mbarriers
    L.es = o;   o = align16(o + sizeof(double) * 4 * 32);
    L.lo = o;   if (comp) o = align16(o + sizeof(uint32_t) * 2 * (size_t)slots);
    L.xs = o;   if (dense_coul) o = align16(o + sizeof(R) * coul_scratch<R>(M * n, !split));
    L.uv = o;   if (coul_smem) o = align16(o + sizeof(R) * 2 * (size_t)n * n);
    if (o < x_end + guard) o = align16(x_end + guard);
    L.ell = o;
    L.total = o;
    return L;
}

// Where a diagonal element's owner leaves the next stage's values: Delta_jj of the partner
// matrix and (split mode) its own diagonal for the partner's records.  In split mode these
// are addresses in the peer CTA's shared memory, written by st.async, which counts the
// bytes on the peer's mbarrier.
template <typename R>
struct PairNext {
    R* dd;                       // this CTA (the partner is matrix m ^ 1); null: not formed by the pass
    uint32_t pdd, pod, pbar;     // peer CTA
    bool fuse;                   // form Delta_jj
    R pulse;
};
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async(uint32_t a, float v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 ::"r"(a), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(uint32_t a, double v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
                 ::"r"(a), "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_peer(uint32_t a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_peer(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
constexpr unsigned ERR_PEER_WAIT = 1u << 5;
// Waits for the phase of `parity`; false after a bounded number of polls.
__device__ __forceinline__ bool peer_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t k = 0; k < (1u << 24); ++k) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// RK accumulators of one element: a register pair in FP32
template <typename R> struct PairAcc { using T = cplx<R>; };
template <> struct PairAcc<float> { using T = uint64_t; };

// Where the neighbours of a slot's elements are, relative to X(i, j) (col: columns j - off,
// j + off, and the same from column j + 1; next: column j + 1): a constant column pitch
// (k_pair), or columns of growing length (k_pair_packed).
template <int NS>
struct PairAddr {
    int pitch;
    const int (&coff)[NS];
    __device__ __forceinline__ int next() const { return pitch; }
    __device__ __forceinline__ int col(int s, int sgn, int e) const { return e * pitch + sgn * coff[s]; }
};

// g = i (X Delta - Delta X) of both elements, FP32 (o0, o1: the elements themselves)
template <int NS, typename ADDR>
__device__ __forceinline__ void pair_sums_f32(const uint64_t* __restrict__ xp, const ADDR ad, uint32_t flags,
                                              const Pattern<float>& pat, uint64_t o0, uint64_t o1, float di, float dj,
                                              float dk, uint64_t& g0, uint64_t& g1)
{
    constexpr int J1 = 2 * NS, SI = 4 * NS;               // flag bits of column j + 1 and of row i
    uint64_t h0 = 0, h1 = 0;                              // g: sums over X(i, k); h: over X(k, j)
    g0 = g1 = 0;
    const uint64_t* xq = xp + ad.next();
    auto terms = [&](auto sc) {
        constexpr int s = decltype(sc)::value;
        constexpr bool L = s == NS - 1;                   // offset 1: the slot's elements are neighbours
        const int o = L ? 1 : pat.off[s];
        f2_add_if<(1u << (2 * s))>(g0, xp[ad.col(s, -1, 0)], flags);
        f2_add_if<(1u << (J1 + 2 * s))>(g1, L ? o0 : xp[ad.col(s, -1, 1)], flags);
        f2_add_if<(1u << (SI + 2 * s))>(h0, xp[-o], flags);
        f2_add_if<(1u << (SI + 2 * s))>(h1, xq[-o], flags);
        f2_add_if<(1u << (2 * s + 1))>(g0, L ? o1 : xp[ad.col(s, 1, 0)], flags);
        f2_add_if<(1u << (J1 + 2 * s + 1))>(g1, xp[ad.col(s, 1, 1)], flags);
        f2_add_if<(1u << (SI + 2 * s + 1))>(h0, xp[o], flags);
        f2_add_if<(1u << (SI + 2 * s + 1))>(h1, xq[o], flags);
    };
    terms(std::integral_constant<int, 0>());
    terms(std::integral_constant<int, 1>());
    if constexpr (NS == 3) terms(std::integral_constant<int, 2>());
    // the diagonal terms once, as X_ij (Delta_jj - Delta_ii): no cancellation
    auto diag_term = [&](uint64_t x, float d, uint64_t t) {
        const cplx<float> u = f2_unpack(x), v = f2_unpack(t);
        return f2_pack(__fmaf_rn(v.re, pat.w, u.re * d), __fmaf_rn(v.im, pat.w, u.im * d));
    };
    g0 = diag_term(o0, dj - di, f2_sub(g0, h0));
    g1 = diag_term(o1, dk - di, f2_sub(g1, h1));
}

// k = -i (X Delta - Delta X) of both elements, FP64: k ascending with the diagonal in
// place, as the oracle sums
template <int NS, typename ADDR>
__device__ __forceinline__ void pair_sums_f64(const cplx<double>* __restrict__ xp, const ADDR ad, uint32_t flags,
                                              const Pattern<double>& pat, double di, double dj, double dk,
                                              cplx<double>& k0, cplx<double>& k1)
{
    constexpr int J1 = 2 * NS, SI = 4 * NS;
    const cplx<double>* xq = xp + ad.next();
    double a0r = 0.0, a0i = 0.0, a1r = 0.0, a1i = 0.0, c0r = 0.0, c0i = 0.0, c1r = 0.0, c1i = 0.0;
    auto add = [&](double& re, double& im, const cplx<double>& x, uint32_t bit) {
        if (flags & bit) { re = __fma_rn(x.re, pat.w, re); im = __fma_rn(x.im, pat.w, im); }
    };
    const cplx<double> o0 = xp[0], o1 = xq[0];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int o = s == NS - 1 ? 1 : pat.off[s];
        add(a0r, a0i, xp[ad.col(s, -1, 0)], 1u << (2 * s));
        add(a1r, a1i, s == NS - 1 ? o0 : xp[ad.col(s, -1, 1)], 1u << (J1 + 2 * s));
        add(c0r, c0i, xp[-o], 1u << (SI + 2 * s));
        add(c1r, c1i, xq[-o], 1u << (SI + 2 * s));
    }
    a0r = __fma_rn(o0.re, dj, a0r); a0i = __fma_rn(o0.im, dj, a0i);
    c0r = __fma_rn(o0.re, di, c0r); c0i = __fma_rn(o0.im, di, c0i);
    a1r = __fma_rn(o1.re, dk, a1r); a1i = __fma_rn(o1.im, dk, a1i);
    c1r = __fma_rn(o1.re, di, c1r); c1i = __fma_rn(o1.im, di, c1i);
#pragma unroll
    for (int s = NS - 1; s >= 0; --s) {
        const int o = s == NS - 1 ? 1 : pat.off[s];
        add(a0r, a0i, s == NS - 1 ? o1 : xp[ad.col(s, 1, 0)], 1u << (2 * s + 1));
        add(a1r, a1i, xp[ad.col(s, 1, 1)], 1u << (J1 + 2 * s + 1));
        add(c0r, c0i, xp[o], 1u << (SI + 2 * s + 1));
        add(c1r, c1i, xq[o], 1u << (SI + 2 * s + 1));
    }
    k0 = {__dsub_rn(a0i, c0i), -__dsub_rn(a0r, c0r)};
    k1 = {__dsub_rn(a1i, c1i), -__dsub_rn(a1r, c1r)};
}

template <typename R, int NT, int SPT, bool SPLIT, int STAGE, int NS, bool DUMP>
__device__ __forceinline__ void pair_pass(const cplx<R>* __restrict__ X, cplx<R>* __restrict__ Xn,
                                          const R* __restrict__ Dd, cplx<R>* __restrict__ rhoS, R* __restrict__ dgn,
                                          const uint32_t (&ix)[SPT], const uint32_t (&fl)[SPT],
                                          typename PairAcc<R>::T (&Ar)[2 * SPT], typename PairAcc<R>::T (&Br)[2 * SPT], R h, int tid,
                                          int n, int RP,
                                          int E, cplx<R>* __restrict__ dump_in, cplx<R>* __restrict__ dump_out,
                                          const DumpMap dm, const PairNext<R>& nx, const DevSys<R>& sys,
                                          const R* __restrict__ sd, uint32_t* __restrict__ loS,
                                          const Pattern<R>& pat)
{
    int coff[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) coff[s] = pat.off[s] * RP;
#pragma unroll
    for (int q = 0; q < SPT; ++q) {
        const int f = tid + q * NT;
        if ((tid & ~31) + q * NT >= E) break;               // this warp's remaining slots are empty
        const uint32_t flags = fl[q];
        const int i = (int)(ix[q] & 1023u), j = (int)((ix[q] >> 10) & 1023u), m = (int)(ix[q] >> 20);
        const int bi = m * n + i, bj = m * n + j;
        const int oij = j * RP + bi, oji = i * RP + bj;
        const bool one = (flags & PAIR_ONE) != 0;
        size_t gi0 = ~size_t(0), gi1 = ~size_t(0);
        if constexpr (DUMP) {
            const int g = dm.split ? m : (m >> 1), s = dm.split ? dm.rank : (m & 1);
            const int b = dm.gbase + g;
            if (b < dm.B && !(flags & PAIR_NONE)) {
                gi0 = ((size_t)b * 2 + s) * dm.ne + (size_t)(cs(j) + i);
                if (!one) gi1 = gi0 + (size_t)(j + 1);      // (i, j + 1)
            }
        }
        cplx<R> r0, r1, x0, x1;
        if constexpr (std::is_same<R, float>::value) {
            const uint64_t* xp = reinterpret_cast<const uint64_t*>(X) + oij;
            const ulonglong2 rr = reinterpret_cast<const ulonglong2*>(rhoS)[f];
            uint64_t &a0 = Ar[2 * q], &b0 = Br[2 * q], &a1 = Ar[2 * q + 1], &b1 = Br[2 * q + 1];
            const uint64_t o0 = f2_stage_input(STAGE, rr.x, a0, b0, h);
            uint64_t o1 = f2_stage_input(STAGE, rr.y, a1, b1, h);
            if (one) o1 = xp[RP];
            uint64_t g0, g1;
            pair_sums_f32<NS>(xp, PairAddr<NS>{RP, coff}, flags, pat, o0, o1, Dd[bi], Dd[bj], Dd[bj + 1], g0, g1);
            if constexpr (STAGE < 3) {
                if (DUMP && STAGE == 0) { r0 = f2_unpack(rr.x); r1 = f2_unpack(rr.y); }
                x0 = f2_unpack(f2_stage(STAGE, rr.x, g0, a0, b0, h));
                x1 = f2_unpack(f2_stage(STAGE, rr.y, g1, a1, b1, h));
            } else {
                uint2 lo = make_uint2(0u, 0u);
                const bool comp = loS != nullptr;
                if (comp) lo = reinterpret_cast<const uint2*>(loS)[f];
                const uint64_t y0 = f2_final(rr.x, g0, b0, h, comp, lo.x), y1 = f2_final(rr.y, g1, b1, h, comp, lo.y);
                const ulonglong2 y = make_ulonglong2(y0, y1);
                if (comp) reinterpret_cast<uint2*>(loS)[f] = lo;
                reinterpret_cast<ulonglong2*>(rhoS)[f] = y;
                x0 = f2_unpack(y.x);
                x1 = f2_unpack(y.y);
            }
        } else {
            // FP64: k ascending with the diagonal in place, as the oracle sums
            cplx<R> k0, k1;
            pair_sums_f64<NS>(X + oij, PairAddr<NS>{RP, coff}, flags, pat, Dd[bi], Dd[bj], Dd[bj + 1], k0, k1);
            r0 = rhoS[2 * f];
            r1 = rhoS[2 * f + 1];
            if (DUMP && STAGE == 0) { x0 = r0; x1 = r1; }
            rk_update<R>(STAGE, k0, h, r0, Ar[2 * q], Br[2 * q], x0);
            rk_update<R>(STAGE, k1, h, r1, Ar[2 * q + 1], Br[2 * q + 1], x1);
            if (STAGE == 3) { rhoS[2 * f] = r0; rhoS[2 * f + 1] = r1; }
        }
        if constexpr (DUMP) {
            if (STAGE == 0) {                              // stage input X1 = rho
                if (gi0 != ~size_t(0)) dump_in[gi0] = r0;
                if (gi1 != ~size_t(0)) dump_in[gi1] = r1;
            }
            if (STAGE < 3) {                               // next stage input
                if (gi0 != ~size_t(0)) dump_out[gi0] = x0;
                if (gi1 != ~size_t(0)) dump_out[gi1] = x1;
            }
        }
        if (flags & PAIR_NONE) continue;
        Xn[oji] = cplx<R>{x0.re, -x0.im};
        Xn[oij] = x0;                         // on the diagonal this second store wins
        if (!one) {
            Xn[oji + 1] = cplx<R>{x1.re, -x1.im};
            Xn[oij + RP] = x1;
        }
        if (i == j) {
            dgn[bi] = x0.re;
            R d = R(0);
            if (nx.fuse) {
                d = sd[i];
                if (sys.coul != 0) {
                    R u = R(0);
                    const R uu = sd[n + i];
                    if (uu != R(0)) u = fmaR<R>(uu, addR<R>(x0.re, sys.shift), u);
                    d = addR<R>(d, u);
                }
                if (sys.has_ext) d = addR<R>(d, sd[2 * n + i]);
                if (sys.n_bins > 0) d = addR<R>(d, mulR<R>(nx.pulse, sd[3 * n + i]));
                if constexpr (!SPLIT) nx.dd[(m ^ 1) * n + i] = d;
            }
            if constexpr (SPLIT) {
                st_async(nx.pdd + (uint32_t)(bi * (int)sizeof(R)), d, nx.pbar);
                st_async(nx.pod + (uint32_t)(bi * (int)sizeof(R)), x0.re, nx.pbar);
            }
        }
    }
}

// SPT: slots (of two elements) per thread.  ResArgs::order holds the slot order
// (pair_slot_order) and ResArgs::nslots their number per matrix.
template <typename R, int NT, int SPT, bool SPLIT, int NS, bool DUMP = false>
__global__ void __launch_bounds__(NT, 512 / NT) k_pair(ResArgs<R> a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = a.sys.n, ne = a.sys.ne;
    const int M = SPLIT ? a.G : 2 * a.G;
    const int RR = M * n;
    const int RP = RR | 1;
    const int E = M * a.nslots;                     // slots in use
    const int DS = RR + 1;                          // stride of the diagonal buffers
    const int XS = n * RP;
    const bool comp = std::is_same<R, float>::value && a.state64 != nullptr;
    const ResLayout<R> L = pair_layout<R>(n, M, NT * SPT, comp, a.pat.off[0], a.sys.ud != nullptr,
                                             a.coul_smem != 0, SPLIT);
    uint32_t* loS = comp ? reinterpret_cast<uint32_t*>(smem + L.lo) : nullptr;
    cplx<R>* Xb = reinterpret_cast<cplx<R>*>(smem + L.x);
    cplx<R>* rhoS = reinterpret_cast<cplx<R>*>(smem + L.rho);
    R* Dd = reinterpret_cast<R*>(smem + L.dd);
    R* dg = reinterpret_cast<R*>(smem + L.dg);
    double* es = reinterpret_cast<double*>(smem + L.es);
    R* scr = reinterpret_cast<R*>(smem + L.xs);
    R* sd = reinterpret_cast<R*>(smem + L.sd);
    const R *ud = a.sys.ud, *vd = a.sys.vd;         // dense Coulomb rows
    if (a.coul_smem) {
        R* uv = reinterpret_cast<R*>(smem + L.uv);
        for (int q = threadIdx.x; q < n * n; q += NT) {
            uv[q] = a.sys.ud[q];
            uv[n * n + q] = a.sys.vd[q];
        }
        ud = uv;
        vd = uv + n * n;
    }
    R* od = Dd + 3 * DS;                            // the other spin's diagonal (split mode), [3][DS] like Dd
    const int tid = threadIdx.x;
    static_assert(NT <= 512, "16 warps per SM at 128 registers");
    const int W = rec_width(n);

    // The two CTAs of a cluster (split mode) meet once per trajectory in a cluster barrier.
    // Within one, a stage ends with a block barrier and a wait for the peer's diagonal,
    // whose values come by st.async into buffer (stage mod 3), counted on that buffer's
    // mbarrier.  Three buffers: the peer can write stage s + 3's values only after it has
    // waited for those this CTA sends in stage s + 1, when it no longer reads stage s's.
    int rank = 0, cid = blockIdx.x, ncl = gridDim.x;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + L.sd + align16(sizeof(R) * 4 * (size_t)n));
    const uint32_t mbar_a = (uint32_t)__cvta_generic_to_shared(mbar);
    uint32_t p_dd = 0, p_od = 0, p_bar = 0;
    if constexpr (SPLIT) {
        cg::cluster_group cl = cg::this_cluster();
        rank = (int)cl.block_rank();
        cid = blockIdx.x >> 1;
        ncl = gridDim.x >> 1;
        p_dd = peer_addr(Dd, rank ^ 1);
        p_od = peer_addr(od, rank ^ 1);
        p_bar = peer_addr(mbar, rank ^ 1);
        if (tid < 3) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_a + 8 * tid) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    uint32_t ph = 0;                                // buffer of the current stage
    uint32_t parity = 0;                            // bit b: the phase buffer b is in
    bool lost = false;                              // a wait gave up
    auto group_bar = [&]() {
        if constexpr (SPLIT) cg::this_cluster().sync(); else __syncthreads();
    };
    auto other_dg = [&](int p, int m) -> const R* {
        if constexpr (SPLIT) return od + ph * DS + m * n;
        else return dg + p * DS + (m ^ 1) * n;
    };

    typename PairAcc<R>::T Ar[2 * SPT], Br[2 * SPT];
    uint32_t ix[SPT], fl[SPT];
#pragma unroll
    for (int q = 0; q < SPT; ++q) {
        const int f = tid + q * NT;
        ix[q] = 0u;
        fl[q] = PAIR_NONE | PAIR_ONE;
        if (f < E) {
            const int m = f / a.nslots;
            const uint32_t p = a.order[f - m * a.nslots];
            if (p == ~0u) continue;
            const uint32_t i = p & 0xffffu, j = (p >> 16) & 0x7fffu;
            const bool one = (p & PAIR_NONE) != 0;
            ix[q] = i | (j << 10) | ((uint32_t)m << 20);
            fl[q] = a.pat.mask[j] | ((one ? 0u : a.pat.mask[j + 1]) << (2 * NS)) | (a.pat.mask[i] << (4 * NS)) |
                    (one ? PAIR_ONE : 0u);
        }
    }
    // packed index and trajectory of a slot's first element; false for slots without a
    // trajectory of this group
    auto place = [&](int q, int gid, size_t& gi) {
        if (fl[q] & PAIR_NONE) return false;
        const int i = (int)(ix[q] & 1023u), j = (int)((ix[q] >> 10) & 1023u), m = (int)(ix[q] >> 20);
        const int g = SPLIT ? m : (m >> 1), s = SPLIT ? rank : (m & 1);
        const int b = gid * a.G + g;
        gi = ((size_t)b * 2 + s) * ne + (size_t)(cs(j) + i);
        return b < a.B;
    };
    double* myslot = a.slots ? a.slots + (size_t)blockIdx.x * a.Tp * W : nullptr;
    // entries no slot writes (the padding row of the odd pitch)
    for (int q = tid; q < 2 * XS; q += NT) Xb[q] = cplx<R>{R(0), R(0)};
    for (int q = tid; q < 2 * DS; q += NT) dg[q] = R(0);
    for (int q = tid; q < 6 * DS; q += NT) Dd[q] = R(0);
    for (int j = tid; j < n; j += NT) {
        sd[j] = a.sys.tdiag[j];
        sd[n + j] = a.udiag ? a.udiag[j] : R(0);
        sd[2 * n + j] = a.sys.ediag[j];
        sd[3 * n + j] = a.sys.proj[j];
    }

    const int ngroups = (a.B + a.G - 1) / a.G;
    group_bar();
    for (int gid = cid; gid < ngroups; gid += ncl) {
#pragma unroll
        for (int q = 0; q < SPT; ++q) {
            const int f = tid + q * NT;
            size_t gi = 0;
            const bool have = place(q, gid, gi);
            const bool one = (fl[q] & PAIR_ONE) != 0;
            const int i = (int)(ix[q] & 1023u), j = (int)((ix[q] >> 10) & 1023u), m = (int)(ix[q] >> 20);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                cplx<R> v = {R(0), R(0)};
                uint32_t lo = 0;
                const size_t ge = e ? gi + (size_t)(j + 1) : gi;
                if (have && !(e && one)) {
                    if (comp) {
                        const cplx<double> x = a.state64[ge];
                        v.re = (R)x.re;
                        v.im = (R)x.im;
                        lo = pack_bf16x2((float)(x.re - (double)v.re), (float)(x.im - (double)v.im));
                    } else {
                        v = a.state[ge];
                    }
                }
                if (!(fl[q] & PAIR_NONE) && !(e && one)) {
                    Xb[i * RP + m * n + j + e] = cplx<R>{v.re, -v.im};
                    Xb[(j + e) * RP + m * n + i] = v;
                    if (i == j + e) {
                        dg[m * n + i] = v.re;
                        if constexpr (SPLIT) st_peer(p_od + (uint32_t)((ph * DS + m * n + i) * (int)sizeof(R)), v.re);
                    }
                }
                rhoS[2 * f + e] = v;
                if (comp) loS[2 * f + e] = lo;
                Ar[2 * q + e] = Br[2 * q + e] = {};
            }
        }
        int cur = 0;
        bool dd_ok = false;                  // Dd[ph] already holds this stage's diagonal
        long gstep = a.step_base;
        group_bar();
        for (int t = a.t_begin; t < a.t_end; ++t) {
            if (a.record) {
                res_record<R, NT, SPLIT>(a, [&](int m, int k, int j) { return Xb[cur * XS + j * RP + m * n + k].re; },
                                         dg + cur * DS, [&](int m) { return other_dg(cur, m); }, es, myslot + (size_t)t * W, gid, rank, tid);
                if (a.whole) {
#pragma unroll
                    for (int q = 0; q < SPT; ++q) {
                        const int f = tid + q * NT;
                        size_t gi = 0;
                        if (!place(q, gid, gi)) continue;
                        const int j = (int)((ix[q] >> 10) & 1023u), m = (int)(ix[q] >> 20);
                        const int s = SPLIT ? rank : (m & 1);
                        const int p = cs(j) + (int)(ix[q] & 1023u);
                        double2* w = a.whole + ((size_t)t * 2 + s) * ne;
                        atomicAdd(&w[p].x, (double)rhoS[2 * f].re);
                        atomicAdd(&w[p].y, (double)rhoS[2 * f].im);
                        if (!(fl[q] & PAIR_ONE)) {
                            atomicAdd(&w[p + j + 1].x, (double)rhoS[2 * f + 1].re);
                            atomicAdd(&w[p + j + 1].y, (double)rhoS[2 * f + 1].im);
                        }
                    }
                }
            }
            const int nsteps = (a.hf && t == a.Tp - 1) ? 0 : a.S;
            for (int st = 0; st < nsteps; ++st, ++gstep) {
#pragma unroll
                for (int stage = 0; stage < 4; ++stage) {
                    R* Dc = Dd + ph * DS;
                    if (!dd_ok) {
                        const R pv = a.sys.n_bins > 0 ? a.ptab[(gstep - a.step_base) * 4 + stage] : R(0);
                        delta_diag_block<R, NT, !SPLIT>(a.sys, ud, vd, Dc, scr, RR, [&](int m) { return dg + cur * DS + m * n; },
                                                [&](int m) { return other_dg(cur, m); }, pv, tid);
                    }
                    // does another stage follow in this launch (possibly after a record)?
                    const bool more = stage < 3 || st + 1 < nsteps ||
                                      (t + 1 < a.t_end && a.S > 0 && !(a.hf && t + 1 == a.Tp - 1));
                    const uint32_t nph = ph == 2 ? 0 : ph + 1;
                    const uint32_t nofs = nph * (uint32_t)(DS * (int)sizeof(R));
                    PairNext<R> nx = {Dd + nph * DS, p_dd + nofs, p_od + nofs, p_bar + 8 * nph, a.udiag != nullptr && more, R(0)};
                    if (nx.fuse && a.sys.n_bins > 0) nx.pulse = a.ptab[(gstep - a.step_base) * 4 + stage + 1];
                    if (SPLIT && tid == 0)
                        asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 s, [%0], %1;\n\t}"
                                     ::"r"(mbar_a + 8 * nph), "r"((uint32_t)(2 * RR * (int)sizeof(R))) : "memory");
                    const cplx<R>* X = Xb + cur * XS;
                    cplx<R>* Xn = Xb + (cur ^ 1) * XS;
                    R* dgn = dg + (cur ^ 1) * DS;
                    cplx<R>* din = nullptr;
                    cplx<R>* dout = nullptr;
                    if (DUMP && a.dump) {
                        din = a.dump + (size_t)(gstep - a.step_base) * 4 * a.dump_count;
                        dout = din + (size_t)(stage + 1) * a.dump_count;
                    }
                    const DumpMap dm = {gid * a.G, rank, a.B, ne, SPLIT ? 1 : 0};
#define FPSG_PAIR_PASS(S_)                                                                                        \
    pair_pass<R, NT, SPT, SPLIT, S_, NS, DUMP>(X, Xn, Dc, rhoS, dgn, ix, fl, Ar, Br, a.h, tid, n, RP, E, din, dout, dm, \
                                               nx, a.sys, sd, loS, a.pat)
                    if (stage == 0) FPSG_PAIR_PASS(0);
                    else if (stage == 1) FPSG_PAIR_PASS(1);
                    else if (stage == 2) FPSG_PAIR_PASS(2);
                    else FPSG_PAIR_PASS(3);
#undef FPSG_PAIR_PASS
                    __syncthreads();
                    if constexpr (SPLIT) {
                        if (!lost && !peer_wait(mbar_a + 8 * nph, (parity >> nph) & 1u)) {
                            lost = true;
                            atomicOr(a.err, ERR_PEER_WAIT);
                        }
                        parity ^= 1u << nph;
                    }
                    cur ^= 1;
                    ph = nph;
                    dd_ok = nx.fuse;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < SPT; ++q) {
            const int f = tid + q * NT;
            size_t gi = 0;
            if (!place(q, gid, gi)) continue;
            const int j = (int)((ix[q] >> 10) & 1023u);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (e && (fl[q] & PAIR_ONE)) continue;
                const size_t ge = e ? gi + (size_t)(j + 1) : gi;
                const cplx<R> v = rhoS[2 * f + e];
                if (comp) {
                    const float2 lo = unpack_bf16x2(loS[2 * f + e]);
                    a.state64[ge] = cplx<double>{(double)v.re + (double)lo.x, (double)v.im + (double)lo.y};
                } else {
                    a.state[ge] = v;
                }
            }
        }
        group_bar();          // the peer has finished with this trajectory too
    }
}

// ------------------------------------------------------------------------------
// k_pair_packed — the pair kernel for one spin matrix per CTA that does not fit twice.
//
// The terms of an upper element reach at most D = off[0] rows below the diagonal, so X is
// kept once, as the upper triangle and the D sub-diagonals, column j in j + D + 1 entries:
//     X(r, c) at C(c) + r,   C(c) = c (c + 2 D + 1) / 2,
// about half of the full matrix, with C(j + o) - C(j) linear in j.  With the state beside it
// that is 194 KB in FP64 at n = 100: a spin on ONE CTA, where k_resident_quad_hp takes two
// (33 four-CTA clusters on 132 SMs; every new element crosses to the sibling through
// distributed shared memory, 16 bytes a cycle; a 460-cycle cluster barrier per stage).  X is
// single-buffered: a pass computes k of every slot into the RK registers, and after a block
// barrier (45 cycles) a second one forms the new stage input from the registers and the
// state and stores it, so no stage output is held across the barrier.  FP64 keeps k1 and k2
// themselves and forms A = k1 - k2 and Bc = k1 + 3 k2 one stage later, by the same
// operations: bit-identical to the oracle.
// 10x10 grid, FP64, 4096 trajectories x 41 steps: 134.7 -> 76 ms
// Spilled per thread, stores / loads in bytes: FP64 with five slots 284 / 364 (n = 100), with four 96
// / 136; FP32 with eight 296 / 68, with eleven (MEMC) 304 / 532; FP64 with three and FP32 with six none.
__host__ __device__ __forceinline__ int packed_col(int c, int D) { return (c * (c + 2 * D + 1)) >> 1; }

// C(j + o) - C(j) = o j + up[s], C(j - o) - C(j) = dn[s] - o j for the offsets o of a
// pattern, and from column j + 1 the column's length more
template <int NS>
struct PackedOffs {
    int o[NS], up[NS], dn[NS];
    __device__ __forceinline__ PackedOffs(const int (&off)[PAT_MAX], int D)
    {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            o[s] = s == NS - 1 ? 1 : off[s];
            up[s] = (o[s] * (o[s] + 2 * D + 1)) >> 1;
            dn[s] = (o[s] * (o[s] - 2 * D - 1)) >> 1;
        }
    }
};
template <int NS>
struct PackedAddr {
    int j, D;
    const PackedOffs<NS>& k;
    __device__ __forceinline__ int next() const { return j + D + 1; }
    __device__ __forceinline__ int col(int s, int sgn, int e) const
    {
        const int o = k.o[s], c = sgn > 0 ? o * j + k.up[s] : k.dn[s] - o * j;
        return e ? c + j + sgn * o + D + 1 : c;
    }
};

template <typename R>
__host__ __device__ __forceinline__ ResLayout<R> packed_layout(int n, int nslots, bool comp, int D, bool dense_coul)
{
    ResLayout<R> L;
    const size_t slots = (size_t)(nslots + 31) / 32 * 32;
    // masked neighbours: C(c) >= -D (D + 1) / 2 for c >= -D, and columns up to n + D; what is
    // there is read and discarded
    const size_t before = sizeof(cplx<R>) * (size_t)(D * (D + 1) / 2 + D + 1);
    const size_t after = sizeof(cplx<R>) * (size_t)(packed_col(n + D + 1, D) + n - packed_col(n, D));
    size_t o = 0;
    L.dd = o;   o = align16(o + sizeof(R) * 6 * ((size_t)n + 1));
    L.dg = o;   o = align16(o + sizeof(R) * ((size_t)n + 1));
    L.sd = o;   o = align16(o + sizeof(R) * 4 * (size_t)n + 32);
    L.es = o;   o = align16(o + sizeof(double) * 4 * 16);
    L.ell = o;  o = align16(o + sizeof(uint32_t) * ((size_t)n + 1));      // the sites' masks
    L.xs = o;   if (dense_coul) o = align16(o + sizeof(R) * coul_scratch<R>(n, false));
    if (o < before) o = align16(before);
    L.x = o;    o = align16(o + sizeof(cplx<R>) * (size_t)(packed_col(n - 1, D) + n));
    const size_t x_end = o;
    L.rho = o;  o = align16(o + sizeof(cplx<R>) * 2 * slots);
    L.lo = o;   if (comp) o = align16(o + sizeof(uint32_t) * 2 * slots);
    if (o < x_end + after) o = align16(x_end + after);
    L.uv = o;
    L.total = o;
    return L;
}

// FP64 stage inputs and accumulators (see rk_update): a, b hold k1, k2 up to stage 3, then
// A + k3 and Bc + 3 k3
__device__ __forceinline__ void packed_acc(int stage, double k, double& a, double& b)
{
    if (stage == 0) { a = k; return; }
    if (stage == 1) { b = k; return; }
    if (stage == 2) {
        const double A = __dsub_rn(a, b), Bc = __dadd_rn(a, __dmul_rn(b, 3.0));
        a = __dadd_rn(A, k);
        b = __dadd_rn(Bc, __dmul_rn(k, 3.0));
        return;
    }
    a = k;
}
__device__ __forceinline__ double packed_next(int stage, double rho, double a, double b, double h)
{
    if (stage == 0) return __dadd_rn(rho, div3_rn(__dmul_rn(a, h)));
    if (stage == 1) return __dadd_rn(rho, __dmul_rn(__dadd_rn(div3_rn(-a), b), h));
    if (stage == 2) return __dadd_rn(rho, __dmul_rn(a, h));
    return __dadd_rn(rho, __dmul_rn(__dmul_rn(__dadd_rn(b, a), h), 0.125));
}

// MEMC: the slots' codes are read again for each pass, from the order table (the next one a
// round ahead) and the sites' masks, instead of held in two registers per slot; that leaves
// room for 11 slots of RK accumulators, FP32 up to n = 144 (12x12 grid, 512 trajectories x 41
// steps: 27.2 ms on two CTAs per spin, 15.4 here).
template <typename R, int NT, int SPT, int NS, bool MEMC = false>
__global__ void __launch_bounds__(NT, 1) k_pair_packed(ResArgs<R> a)
{
    static_assert(NT == 512, "packed_layout has room for 16 warps' energy partials");
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool kFloat = std::is_same<R, float>::value;
    const int n = a.sys.n, ne = a.sys.ne, D = a.pat.off[0];
    const int E = a.nslots, DS = n + 1;
    const bool comp = kFloat && a.state64 != nullptr;
    const ResLayout<R> L = packed_layout<R>(n, a.nslots, comp, D, a.sys.ud != nullptr);
    cplx<R>* X = reinterpret_cast<cplx<R>*>(smem + L.x);
    cplx<R>* rhoS = reinterpret_cast<cplx<R>*>(smem + L.rho);
    uint32_t* loS = reinterpret_cast<uint32_t*>(smem + L.lo);
    R* Dd = reinterpret_cast<R*>(smem + L.dd);      // [3][DS], and the other spin's diagonal [3][DS]
    R* od = Dd + 3 * DS;
    R* dg = reinterpret_cast<R*>(smem + L.dg);
    R* sd = reinterpret_cast<R*>(smem + L.sd);
    double* es = reinterpret_cast<double*>(smem + L.es);
    R* scr = reinterpret_cast<R*>(smem + L.xs);
    const int tid = threadIdx.x;
    const int W = rec_width(n);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
    // the exchange of diagonals with the other spin's CTA is k_pair's
    const uint32_t mbar_a = (uint32_t)__cvta_generic_to_shared(smem + L.sd + align16(sizeof(R) * 4 * (size_t)n));
    const uint32_t p_dd = peer_addr(Dd, rank ^ 1), p_od = peer_addr(od, rank ^ 1), p_bar = peer_addr(smem + L.sd + align16(sizeof(R) * 4 * (size_t)n), rank ^ 1);
    if (tid < 3) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_a + 8 * tid) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    uint32_t ph = 0, parity = 0;
    bool lost = false;
    const PackedOffs<NS> offs(a.pat.off, D);

    typename PairAcc<R>::T Ar[2 * SPT], Br[2 * SPT];
    uint32_t* mk = reinterpret_cast<uint32_t*>(smem + L.ell);
    for (int j = tid; j <= n; j += NT) mk[j] = j < n ? a.pat.mask[j] : 0u;
    __syncthreads();
    struct Slot {
        int i, j;
        uint32_t fl;                         // as in k_pair
    };
    auto order_at = [&](int f) { return f < E ? __ldg(a.order + f) : ~0u; };
    auto slot_of = [&](uint32_t p) -> Slot {
        if (p == ~0u) return Slot{0, 0, PAIR_NONE | PAIR_ONE};
        const int i = (int)(p & 0xffffu), j = (int)((p >> 16) & 0x7fffu);
        const bool one = (p & PAIR_NONE) != 0;
        return Slot{i, j, mk[j] | ((one ? 0u : mk[j + 1]) << (2 * NS)) | (mk[i] << (4 * NS)) | (one ? PAIR_ONE : 0u)};
    };
    uint32_t ix[MEMC ? 1 : SPT], fl[MEMC ? 1 : SPT];
    if constexpr (!MEMC) {
#pragma unroll
        for (int q = 0; q < SPT; ++q) {
            const Slot s = slot_of(order_at(tid + q * NT));
            ix[q] = (uint32_t)s.i | ((uint32_t)s.j << 10);
            fl[q] = s.fl;
        }
    }
    // slot q; `next` carries the following one's code (MEMC)
    auto get = [&](int q, uint32_t& next) -> Slot {
        if constexpr (MEMC) {
            const uint32_t p = next;
            next = order_at(tid + (q + 1) * NT);
            return slot_of(p);
        } else {
            return Slot{(int)(ix[q] & 1023u), (int)(ix[q] >> 10), fl[q]};
        }
    };
    auto first = [&]() -> uint32_t { if constexpr (MEMC) return order_at(tid); else return 0u; };
    for (int q = tid; q < 6 * DS; q += NT) Dd[q] = R(0);
    for (int j = tid; j < n; j += NT) {
        sd[j] = a.sys.tdiag[j];
        sd[n + j] = a.udiag ? a.udiag[j] : R(0);
        sd[2 * n + j] = a.sys.ediag[j];
        sd[3 * n + j] = a.sys.proj[j];
    }
    for (int q = tid; q < packed_col(n - 1, D) + n; q += NT) X[q] = cplx<R>{R(0), R(0)};   // rows past n - 1
    double* myslot = a.slots ? a.slots + (size_t)blockIdx.x * a.Tp * W : nullptr;
    cl.sync();
    for (int b = cid; b < a.B; b += ncl) {
        const size_t base = ((size_t)b * 2 + rank) * ne;
        uint32_t nc = first();
#pragma unroll
        for (int q = 0; q < SPT; ++q) {
            Ar[2 * q] = Br[2 * q] = Ar[2 * q + 1] = Br[2 * q + 1] = {};
            if ((tid & ~31) + q * NT >= E) continue;
            const Slot sl = get(q, nc);
            const int f = tid + q * NT, i = sl.i, j = sl.j;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                cplx<R> v = {R(0), R(0)};
                uint32_t lo = 0;
                if (!(sl.fl & PAIR_NONE) && !(e && (sl.fl & PAIR_ONE))) {
                    const int c = j + e;
                    if (comp) {
                        const cplx<double> x = a.state64[base + cs(c) + i];
                        v.re = (R)x.re;
                        v.im = (R)x.im;
                        lo = pack_bf16x2((float)(x.re - (double)v.re), (float)(x.im - (double)v.im));
                    } else {
                        v = a.state[base + cs(c) + i];
                    }
                    if (c - i <= D) X[packed_col(i, D) + c] = cplx<R>{v.re, -v.im};
                    X[packed_col(c, D) + i] = v;
                    if (i == c) {
                        dg[i] = v.re;
                        st_peer(p_od + (uint32_t)((ph * DS + i) * (int)sizeof(R)), v.re);
                    }
                }
                rhoS[2 * f + e] = v;
                if (comp) loS[2 * f + e] = lo;
            }
        }
        bool dd_ok = false;                  // Dd[ph] already holds this stage's diagonal
        long gstep = a.step_base;
        cl.sync();
        for (int t = a.t_begin; t < a.t_end; ++t) {
            if (a.record) {
                res_record<R, NT, true>(a, [&](int, int k, int j) { return X[packed_col(j, D) + k].re; }, dg,
                                        [&](int) { return od + ph * DS; }, es, myslot + (size_t)t * W, b, rank, tid);
                if (a.whole) {
                    uint32_t nc = first();
#pragma unroll
                    for (int q = 0; q < SPT; ++q) {
                        if ((tid & ~31) + q * NT >= E) break;
                        const Slot sl = get(q, nc);
                        if (sl.fl & PAIR_NONE) continue;
                        const int f = tid + q * NT, i = sl.i, j = sl.j;
                        double2* w = a.whole + ((size_t)t * 2 + rank) * ne;
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (e && (sl.fl & PAIR_ONE)) continue;
                            atomicAdd(&w[cs(j + e) + i].x, (double)rhoS[2 * f + e].re);
                            atomicAdd(&w[cs(j + e) + i].y, (double)rhoS[2 * f + e].im);
                        }
                    }
                }
            }
            const int nsteps = (a.hf && t == a.Tp - 1) ? 0 : a.S;
            for (int st = 0; st < nsteps; ++st, ++gstep) {
#pragma unroll 1
                for (int stage = 0; stage < 4; ++stage) {
                    R* Dc = Dd + ph * DS;
                    if (!dd_ok) {
                        const R pv = a.sys.n_bins > 0 ? a.ptab[(gstep - a.step_base) * 4 + stage] : R(0);
                        delta_diag_block<R, NT, false>(a.sys, a.sys.ud, a.sys.vd, Dc, scr, n, [&](int) { return dg; },
                                                       [&](int) { return od + ph * DS; }, pv, tid);
                    }
                    const bool more = stage < 3 || st + 1 < nsteps ||
                                      (t + 1 < a.t_end && a.S > 0 && !(a.hf && t + 1 == a.Tp - 1));
                    const bool fuse = a.udiag != nullptr && more;
                    const R pvn = fuse && a.sys.n_bins > 0 ? a.ptab[(gstep - a.step_base) * 4 + stage + 1] : R(0);
                    const uint32_t nph = ph == 2 ? 0 : ph + 1;
                    if (tid == 0)
                        asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 s, [%0], %1;\n\t}"
                                     ::"r"(mbar_a + 8 * nph), "r"((uint32_t)(2 * n * (int)sizeof(R))) : "memory");
                    // k of every slot
                    uint32_t nc = first();
#pragma unroll
                    for (int q = 0; q < SPT; ++q) {
                        if ((tid & ~31) + q * NT >= E) break;       // this warp's remaining slots are empty
                        const Slot sl = get(q, nc);
                        const int i = sl.i, j = sl.j;
                        const PackedAddr<NS> ad = {j, D, offs};
                        const int xo = packed_col(j, D) + i;
                        if constexpr (kFloat) {
                            const uint64_t* xp = reinterpret_cast<const uint64_t*>(X) + xo;
                            const uint64_t o0 = xp[0], o1 = xp[ad.next()];
                            uint64_t g0, g1;
                            pair_sums_f32<NS>(xp, ad, sl.fl, a.pat, o0, o1, Dc[i], Dc[j], Dc[j + 1], g0, g1);
                            if (stage == 0) { Ar[2 * q] = g0; Ar[2 * q + 1] = g1; }
                            else if (stage == 1) { Br[2 * q] = g0; Br[2 * q + 1] = g1; }
                            else if (stage == 2) {
                                f2_stage(2, 0, g0, Ar[2 * q], Br[2 * q], a.h);
                                f2_stage(2, 0, g1, Ar[2 * q + 1], Br[2 * q + 1], a.h);
                            } else { Ar[2 * q] = g0; Ar[2 * q + 1] = g1; }
                        } else {
                            cplx<R> k0, k1;
                            pair_sums_f64<NS>(X + xo, ad, sl.fl, a.pat, Dc[i], Dc[j], Dc[j + 1], k0, k1);
                            packed_acc(stage, k0.re, Ar[2 * q].re, Br[2 * q].re);
                            packed_acc(stage, k0.im, Ar[2 * q].im, Br[2 * q].im);
                            packed_acc(stage, k1.re, Ar[2 * q + 1].re, Br[2 * q + 1].re);
                            packed_acc(stage, k1.im, Ar[2 * q + 1].im, Br[2 * q + 1].im);
                        }
                    }
                    nc = first();
                    __syncthreads();         // every thread is done reading X
#pragma unroll
                    for (int q = 0; q < SPT; ++q) {
                        const int f = tid + q * NT;
                        if ((tid & ~31) + q * NT >= E) break;
                        const Slot sl = get(q, nc);
                        const int i = sl.i, j = sl.j;
                        cplx<R> x0, x1;
                        if constexpr (kFloat) {
                            const ulonglong2 rr = reinterpret_cast<const ulonglong2*>(rhoS)[f];
                            ulonglong2 y;
                            if (stage < 3) {
                                y.x = f2_stage_input(stage + 1, rr.x, Ar[2 * q], Br[2 * q], a.h);
                                y.y = f2_stage_input(stage + 1, rr.y, Ar[2 * q + 1], Br[2 * q + 1], a.h);
                            } else {
                                uint2 lo = make_uint2(0u, 0u);
                                if (comp) lo = reinterpret_cast<const uint2*>(loS)[f];
                                y.x = f2_final(rr.x, Ar[2 * q], Br[2 * q], a.h, comp, lo.x);
                                y.y = f2_final(rr.y, Ar[2 * q + 1], Br[2 * q + 1], a.h, comp, lo.y);
                                if (comp) reinterpret_cast<uint2*>(loS)[f] = lo;
                                reinterpret_cast<ulonglong2*>(rhoS)[f] = y;
                            }
                            x0 = f2_unpack(y.x);
                            x1 = f2_unpack(y.y);
                        } else {
                            const cplx<R> r0 = rhoS[2 * f], r1 = rhoS[2 * f + 1];
                            x0.re = packed_next(stage, r0.re, Ar[2 * q].re, Br[2 * q].re, a.h);
                            x0.im = packed_next(stage, r0.im, Ar[2 * q].im, Br[2 * q].im, a.h);
                            x1.re = packed_next(stage, r1.re, Ar[2 * q + 1].re, Br[2 * q + 1].re, a.h);
                            x1.im = packed_next(stage, r1.im, Ar[2 * q + 1].im, Br[2 * q + 1].im, a.h);
                            if (stage == 3) { rhoS[2 * f] = x0; rhoS[2 * f + 1] = x1; }
                        }
                        if (sl.fl & PAIR_NONE) continue;
                        const int cj = packed_col(j, D), ci = packed_col(i, D);
                        if (j - i <= D) X[ci + j] = cplx<R>{x0.re, -x0.im};
                        X[cj + i] = x0;                       // on the diagonal this second store wins
                        if (!(sl.fl & PAIR_ONE)) {
                            if (j + 1 - i <= D) X[ci + j + 1] = cplx<R>{x1.re, -x1.im};
                            X[cj + j + D + 1 + i] = x1;
                        }
                        if (i == j) {
                            dg[i] = x0.re;
                            R d = R(0);
                            if (fuse) {
                                // Delta_ii of the other spin for the next stage (on-site U only)
                                d = sd[i];
                                if (a.sys.coul != 0) {
                                    R u = R(0);
                                    const R uu = sd[n + i];
                                    if (uu != R(0)) u = fmaR<R>(uu, addR<R>(x0.re, a.sys.shift), u);
                                    d = addR<R>(d, u);
                                }
                                if (a.sys.has_ext) d = addR<R>(d, sd[2 * n + i]);
                                if (a.sys.n_bins > 0) d = addR<R>(d, mulR<R>(pvn, sd[3 * n + i]));
                            }
                            const uint32_t o = (nph * DS + i) * (uint32_t)sizeof(R);
                            st_async(p_dd + o, d, p_bar + 8 * nph);
                            st_async(p_od + o, x0.re, p_bar + 8 * nph);
                        }
                    }
                    __syncthreads();
                    if (!lost && !peer_wait(mbar_a + 8 * nph, (parity >> nph) & 1u)) {
                        lost = true;
                        atomicOr(a.err, ERR_PEER_WAIT);
                    }
                    parity ^= 1u << nph;
                    ph = nph;
                    dd_ok = fuse;
                }
            }
        }
        nc = first();
#pragma unroll
        for (int q = 0; q < SPT; ++q) {
            if ((tid & ~31) + q * NT >= E) break;
            const Slot sl = get(q, nc);
            if (sl.fl & PAIR_NONE) continue;
            const int f = tid + q * NT, i = sl.i, j = sl.j;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                if (e && (sl.fl & PAIR_ONE)) continue;
                const cplx<R> v = rhoS[2 * f + e];
                const size_t ge = base + cs(j + e) + i;
                if (comp) {
                    const float2 l = unpack_bf16x2(loS[2 * f + e]);
                    a.state64[ge] = cplx<double>{(double)v.re + (double)l.x, (double)v.im + (double)l.y};
                } else {
                    a.state[ge] = v;
                }
            }
        }
        cl.sync();            // the other CTA has finished with this trajectory too
    }
}

}  // namespace fpsg
