// fpsg_fock.cuh — Hartree-Fock with a same-spin V (the Fock term), one trajectory per
// cluster.
//
// Delta = tM + diag(U n_other + V n_same) - N o V (+ potential, pulse) is dense, complex
// and different for every matrix and stage (src/FHHFSolver.cpp:575-608), so a stage is a
// dense complex commutator, 16 n^3 FP64 multiply-adds per spin, of usually ONE trajectory.
// k_fock_stage gives each spin one CTA and reads X and Delta from global memory: the whole
// GPU waits for two CTAs.  Here a cluster of 2 CPS CTAs (8 per spin) runs the trajectory for
// a whole time window: every CTA holds its spin's full X (and Delta, where both fit) in
// shared memory and computes every CPS-th 32-slot chunk of the upper triangle; its new
// elements go to the spin's other CTAs through distributed shared memory.
//
// A slot is two elements (i, j), (i, j + 1) (pair_slot_order): per k, two 16-byte lane
// reads (X_ik, Delta_ik) and four broadcasts (Delta_kj, X_kj of both columns, by component)
// feed 16 multiply-adds, 16 shared-memory wavefronts instead of 24 for two separate ones.  The
// chains over k run in ascending order, each complex multiply-add as four fused ones in the
// order of cmaddR: FP64 results are the oracle's to the bit.  A stage of the 8x8 grid takes
// 20 K cycles: the sums over k 7 to 10 K (one or two busy warps per scheduler, about 110
// cycles per k and warp), Delta 3.3 K, the Hartree chains 2 K, the snapshot record 2.4 K,
// sending the new elements 2.5 K (distributed shared memory takes 16 bytes a cycle), the
// two cluster barriers 2.4 K.  800 stages: 86.2 -> 8.3 ms.
#pragma once
#include "fpsg_kernels.cuh"
#include "fpsg_pair.cuh"

namespace fpsg {

constexpr int FOCK_NT = 512;

template <typename R>
struct FockRunArgs {
    DevSys<R> sys;
    const R *tMf, *Uf, *Vf, *extf;     // dense real parts [n][n] (symmetric)
    int uv_same;                       // U and V agree off the diagonal
    int ext_diag;                      // the potential is diagonal
    cplx<R>* state;                    // [B][2][ne]
    cplx<R>* Dg;                       // [2 B][n][P] Delta in global memory; null: in shared memory
    int B, cps;                        // trajectories; CTAs per spin
    R h;
    const R* ptab;                     // pulse value per (step, stage) from the launch's first step
    int t_begin, t_end, S, Tp;
    int record, do_en, do_e1, do_e2, hf;
    double* diagbuf;                   // [Tp][B][2][n]
    double* ebuf;                      // [Tp][B][2][4]
    double2* whole;                    // [Tp][2][ne] or null
    const uint32_t* order;             // pair_slot_order
    int nslots;
    unsigned* err;
};

template <typename R>
struct FockLayout {
    size_t x, d, od, u, es, sd, tv, ij, total;
};
template <typename R>
__host__ __device__ __forceinline__ FockLayout<R> fock_layout(int n, bool d_smem, bool tv_smem)
{
    const size_t P = (size_t)(n | 1);
    FockLayout<R> L;
    size_t o = 0;
    L.x = o;  o = align16(o + sizeof(cplx<R>) * (size_t)n * P);
    L.d = o;  if (d_smem) o = align16(o + sizeof(cplx<R>) * (size_t)n * P);
    L.od = o; o = align16(o + sizeof(R) * (size_t)n);           // the other spin's diagonal
    L.u = o;  o = align16(o + sizeof(R) * 2 * (size_t)n);       // Hartree sums of U and V
    L.es = o; o = align16(o + sizeof(double) * 32);
    L.sd = o; o = align16(o + sizeof(R) * 2 * (size_t)n);       // U_jj, extPot_jj
    L.tv = o; if (tv_smem) o = align16(o + sizeof(R) * 2 * (size_t)n * n);
    L.ij = o; if (tv_smem) o = align16(o + sizeof(uint32_t) * (size_t)(n * (n + 1) / 2));
    L.total = o;
    return L;
}

__device__ __forceinline__ void st_peer(uint32_t a, cplx<double> v)
{
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.re), "d"(v.im) : "memory");
}
__device__ __forceinline__ void st_peer(uint32_t a, cplx<float> v)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.re), "f"(v.im) : "memory");
}

// Complex numbers from shared memory by 32-bit address: whole (lanes reading consecutive
// ones), or by component for addresses all lanes share (an 8-byte broadcast is one
// wavefront, a 16-byte one four).  The loads are asm that the compiler may move (as volatile
// ones each waited for the one before: 12 to 21 K cycles for a sweep over k of 7 to 10), so
// what orders them is data: every address derives from a base taken by after_barrier behind
// the barrier that publishes the contents, and before_barrier takes what was formed from them
// ahead of the barrier that lets the contents change.
__device__ __forceinline__ uint32_t after_barrier(const void* p)
{
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("" : "+r"(a)::"memory");
    return a;
}
__device__ __forceinline__ void before_barrier(cplx<double>& v) { asm volatile("" : "+d"(v.re), "+d"(v.im)::"memory"); }
__device__ __forceinline__ void before_barrier(cplx<float>& v) { asm volatile("" : "+f"(v.re), "+f"(v.im)::"memory"); }
__device__ __forceinline__ void lds_cplx(cplx<double>& v, uint32_t a)
{
    asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.re), "=d"(v.im) : "r"(a));
}
__device__ __forceinline__ void lds_cplx(cplx<float>& v, uint32_t a)
{
    asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.re), "=f"(v.im) : "r"(a));
}
__device__ __forceinline__ void lds_parts(cplx<double>& v, uint32_t a)
{
    asm("ld.shared.f64 %0, [%1];" : "=d"(v.re) : "r"(a));
    asm("ld.shared.f64 %0, [%1+8];" : "=d"(v.im) : "r"(a));
}
__device__ __forceinline__ void lds_parts(cplx<float>& v, uint32_t a) { lds_cplx(v, a); }

// DSMEM: Delta in shared memory; TVSMEM: tM, V and the elements' indices too
template <typename R, bool DSMEM, bool TVSMEM>
__global__ void __launch_bounds__(FOCK_NT, 1) k_fock_run(FockRunArgs<R> a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = a.sys.n, ne = a.sys.ne, P = n | 1, CPS = a.cps;
    const FockLayout<R> L = fock_layout<R>(n, DSMEM, TVSMEM);
    cplx<R>* X = reinterpret_cast<cplx<R>*>(smem + L.x);         // X(i, k) at k * P + i
    R* od = reinterpret_cast<R*>(smem + L.od);
    R* hs = reinterpret_cast<R*>(smem + L.u);                    // [2][n]
    double* es = reinterpret_cast<double*>(smem + L.es);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int spin = rank / CPS, part = rank - spin * CPS;
    const int cid = blockIdx.x / (2 * CPS), ncl = gridDim.x / (2 * CPS);
    const DevSys<R>& s = a.sys;
    R* sd = reinterpret_cast<R*>(smem + L.sd);
    for (int k = tid; k < n; k += FOCK_NT) {
        sd[k] = a.Uf[(size_t)k * n + k];
        sd[n + k] = a.extf[(size_t)k * n + k];
    }
    R* tv = reinterpret_cast<R*>(smem + L.tv);
    if constexpr (TVSMEM)
        for (int q = tid; q < n * n; q += FOCK_NT) {
            tv[q] = a.tMf[q];
            tv[n * n + q] = a.Vf[q];
        }
    uint32_t* ijs = reinterpret_cast<uint32_t*>(smem + L.ij);
    if constexpr (TVSMEM)
        for (int p = tid; p < ne; p += FOCK_NT) ijs[p] = s.pij[p];
    auto t_at = [&](int q) -> R { if constexpr (TVSMEM) return tv[q]; else return a.tMf[q]; };
    auto v_at = [&](int q) -> R { if constexpr (TVSMEM) return tv[n * n + q]; else return a.Vf[q]; };

    // this thread's slot: chunk part + CPS * warp of 32 slots
    const int f = (part + CPS * warp) * 32 + lane;
    const uint32_t code = f < a.nslots ? a.order[f] : ~0u;
    const bool have = code != ~0u;
    const int i = have ? (int)(code & 0xffffu) : 0, j = have ? (int)((code >> 16) & 0x7fffu) : 0;
    const bool two = have && !(code & PAIR_NONE);
    const int j1 = two ? j + 1 : j;
    const bool busy = (part + CPS * warp) * 32 < a.nslots;       // this warp has slots

    for (int b = cid; b < a.B; b += ncl) {
        const size_t base = ((size_t)b * 2 + spin) * ne;
        cplx<R>* Dm = DSMEM ? reinterpret_cast<cplx<R>*>(smem + L.d)
                            : a.Dg + ((size_t)b * 2 + spin) * (size_t)n * P;
        const cplx<R> z = {R(0), R(0)};
        for (int p = tid; p < ne; p += FOCK_NT) {
            const uint32_t ij = s.pij[p];
            X[(ij >> 16) * P + (ij & 0xffffu)] = a.state[base + p];
        }
        for (int k = tid; k < n; k += FOCK_NT) od[k] = a.state[((size_t)b * 2 + (spin ^ 1)) * ne + cs(k) + k].re;
        cplx<R> r0 = have ? a.state[base + cs(j) + i] : z, r1 = two ? a.state[base + cs(j1) + i] : z;
        cplx<R> A0 = z, A1 = z, B0 = z, B1 = z;
        long g = 0;                                              // (step, stage) of the launch
        __syncthreads();
        for (int t = a.t_begin; t < a.t_end; ++t) {
            const int nsteps = (a.hf && t == a.Tp - 1) ? 0 : a.S;
            for (int st = 0; st < nsteps || st == 0; ++st) {
                for (int stage = 0; stage < 4; ++stage, ++g) {
                    if (a.record && st == 0 && stage == 0) {
                        double* db = a.diagbuf + (((size_t)t * a.B + b) * 2 + spin) * n;
                        if (part == 0)
                            for (int k = tid; k < n; k += FOCK_NT) {
                                const double d = (double)X[k * P + k].re;
                                if (!isfinite(d)) atomicOr(a.err, 1u);
                                db[k] = d;
                            }
                        // energy rows (see energy_partials; the exchange term is -V_jk |N_jk|^2 / 2), row c on
                        // the spin's CTA c mod CPS
                        for (int c = 0; c < 4 && a.do_en; ++c) {
                            if (c % CPS != part) continue;
                            double e = 0.0;
                            if (c == 0 || (c == 3 && s.has_ext) || (c == 1 && a.do_e1 && spin == 0) || (c == 2 && a.do_e2))
#pragma unroll 2
                                for (int p = tid; p < ne; p += FOCK_NT) {        // both triangles from the upper one
                                    const uint32_t ij = TVSMEM ? ijs[p] : s.pij[p];
                                    const int x = (int)(ij & 0xffffu), y = (int)(ij >> 16), q = y * n + x;
                                    const cplx<R> v = X[y * P + x];
                                    const double w = x == y ? 1.0 : 2.0;
                                    if (c == 0) e += w * ((double)v.re * (double)t_at(q));
                                    else if (c == 3) e += w * ((double)v.re * (double)(a.ext_diag ? (x == y ? sd[n + x] : R(0)) : a.extf[q]));
                                    else {
                                        const double ny = (double)X[y * P + y].re, nx = (double)X[x * P + x].re;
                                        if (c == 1) {
                                            const R u = !a.uv_same ? a.Uf[q] : x == y ? sd[x] : v_at(q);
                                            e += w * 0.5 * (double)u * (ny * (double)od[x] + (double)od[y] * nx);
                                        } else {
                                            e += w * 0.5 * (double)v_at(q) *
                                                 (ny * nx - ((double)v.re * (double)v.re + (double)v.im * (double)v.im));
                                        }
                                    }
                                }
                            e = warp_sum(e);
                            if (lane == 0) es[warp] = e;
                            __syncthreads();
                            if (tid == 0) {
                                double v = 0.0;
                                for (int q = 0; q < FOCK_NT / 32; ++q) v += es[q];
                                a.ebuf[(((size_t)t * a.B + b) * 2 + spin) * 4 + c] = v;
                            }
                            __syncthreads();
                        }
                        if (a.whole && have) {
                            double2* w = a.whole + ((size_t)t * 2 + spin) * ne;
                            atomicAdd(&w[cs(j) + i].x, (double)r0.re);
                            atomicAdd(&w[cs(j) + i].y, (double)r0.im);
                            if (two) {
                                atomicAdd(&w[cs(j1) + i].x, (double)r1.re);
                                atomicAdd(&w[cs(j1) + i].y, (double)r1.im);
                            }
                        }
                    }
                    if (nsteps == 0) { st = 1; break; }
                    // Hartree sums, ascending k: U n_other on threads 0 .. n-1, V n_same on the next n
                    for (int q = tid; q < 2 * n; q += FOCK_NT) {
                        const bool vt = q >= n;
                        const int jj = vt ? q - n : q;
                        R acc = R(0);
                        if (vt) {
#pragma unroll 8
                            for (int k = 0; k < n; ++k) acc = fmaR<R>(v_at(k * n + jj), X[k * P + k].re, acc);
                        } else if (a.uv_same) {
                            const R wd = sd[jj];
#pragma unroll 8
                            for (int k = 0; k < n; ++k) {
                                const R w = v_at(k * n + jj);
                                acc = fmaR<R>(k == jj ? wd : w, addR<R>(od[k], s.shift), acc);
                            }
                        } else {
#pragma unroll 16
                            for (int k = 0; k < n; ++k) acc = fmaR<R>(a.Uf[(size_t)k * n + jj], addR<R>(od[k], s.shift), acc);
                        }
                        hs[q] = acc;
                    }
                    __syncthreads();
                    // Delta from the upper triangle of X, additions in the oracle's order (its lower
                    // triangle is the conjugate to the bit), and the lower triangle of X; with Delta in
                    // global memory each CTA of the spin writes its share of the columns
                    const R pulse = s.n_bins > 0 ? a.ptab[g] : R(0);
#pragma unroll 2
                    for (int p = tid; p < ne; p += FOCK_NT) {
                        const uint32_t ij = TVSMEM ? ijs[p] : s.pij[p];
                        const int r = (int)(ij & 0xffffu), c = (int)(ij >> 16), q = c * n + r;
                        const cplx<R> x = X[c * P + r];
                        const bool diag = r == c;
                        if (!diag) X[r * P + c] = cplx<R>{x.re, -x.im};
                        if (!DSMEM && (c % CPS) != part) continue;
                        const R vij = v_at(q);
                        cplx<R> d = {t_at(q), R(0)};
                        if (diag && s.coul != 0) d.re = addR<R>(d.re, hs[c]);
                        const R nvr = mulR<R>(x.re, vij), nvi = mulR<R>(x.im, vij);
                        d.re = addR<R>(d.re, diag ? subR<R>(hs[n + c], nvr) : subR<R>(R(0), nvr));
                        d.im = addR<R>(d.im, subR<R>(R(0), nvi));
                        if (s.has_ext) d.re = addR<R>(d.re, a.ext_diag ? (diag ? sd[n + c] : R(0)) : a.extf[q]);
                        if (diag && s.n_bins > 0) d.re = addR<R>(d.re, mulR<R>(pulse, s.proj[c]));
                        Dm[c * P + r] = d;
                        if (!diag) Dm[r * P + c] = cplx<R>{d.re, -d.im};
                    }
                    if constexpr (DSMEM) __syncthreads();
                    else { __threadfence(); cl.sync(); }        // the other CTAs' columns
                    cplx<R> x0 = z, x1 = z;
                    if (busy) {
                        cplx<R> a0 = z, a1 = z, b0 = z, b1 = z;
                        // the operands of the next k are on their way while this one's 16 multiply-adds
                        // run: a CTA has one or two busy warps per scheduler
                        if constexpr (DSMEM) {
                            const uint32_t sz = (uint32_t)sizeof(cplx<R>), row = (uint32_t)P * sz;
                            const uint32_t Xa = after_barrier(X), Da = after_barrier(Dm);
                            uint32_t xi = Xa + i * sz, ei = Da + i * sz;
                            uint32_t yj = Xa + j * row, yk = Xa + j1 * row, dj = Da + j * row, dk = Da + j1 * row;
                            cplx<R> x, e, d0, d1, y0, y1;
                            lds_cplx(x, xi); lds_cplx(e, ei);
                            lds_parts(d0, dj); lds_parts(d1, dk); lds_parts(y0, yj); lds_parts(y1, yk);
#pragma unroll 4
                            for (int k = 1; k < n; ++k) {
                                xi += row; ei += row;
                                const cplx<R> cx = x, ce = e, c0 = d0, c1 = d1, v0 = y0, v1 = y1;
                                lds_cplx(x, xi); lds_cplx(e, ei);
                                lds_parts(d0, dj + k * sz); lds_parts(d1, dk + k * sz);
                                lds_parts(y0, yj + k * sz); lds_parts(y1, yk + k * sz);
                                cmaddR<R>(a0.re, a0.im, cx, c0);
                                cmaddR<R>(a1.re, a1.im, cx, c1);
                                cmaddR<R>(b0.re, b0.im, v0, ce);
                                cmaddR<R>(b1.re, b1.im, v1, ce);
                            }
                            cmaddR<R>(a0.re, a0.im, x, d0);
                            cmaddR<R>(a1.re, a1.im, x, d1);
                            cmaddR<R>(b0.re, b0.im, y0, e);
                            cmaddR<R>(b1.re, b1.im, y1, e);
                            before_barrier(a0); before_barrier(a1); before_barrier(b0); before_barrier(b1);
                        } else {
                            auto ld = [](const cplx<R>* p) -> cplx<R> {     // written by other SMs: not from L1
                                using V = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
                                const V v = __ldcg(reinterpret_cast<const V*>(p));
                                return cplx<R>{(R)v.x, (R)v.y};
                            };
                            const cplx<R> *dj = Dm + j * P, *dk = Dm + j1 * P, *yj = X + j * P, *yk = X + j1 * P;
#pragma unroll 2
                            for (int k = 0; k < n; ++k) {
                                const cplx<R> x = X[k * P + i], e = ld(Dm + k * P + i);
                                cmaddR<R>(a0.re, a0.im, x, ld(dj + k));
                                cmaddR<R>(a1.re, a1.im, x, ld(dk + k));
                                cmaddR<R>(b0.re, b0.im, yj[k], e);
                                cmaddR<R>(b1.re, b1.im, yk[k], e);
                            }
                        }
                        const cplx<R> k0 = {subR<R>(a0.im, b0.im), -subR<R>(a0.re, b0.re)};
                        const cplx<R> k1 = {subR<R>(a1.im, b1.im), -subR<R>(a1.re, b1.re)};
                        if (stage == 0) { rk_update<R>(0, k0, a.h, r0, A0, B0, x0); rk_update<R>(0, k1, a.h, r1, A1, B1, x1); }
                        else if (stage == 1) { rk_update<R>(1, k0, a.h, r0, A0, B0, x0); rk_update<R>(1, k1, a.h, r1, A1, B1, x1); }
                        else if (stage == 2) { rk_update<R>(2, k0, a.h, r0, A0, B0, x0); rk_update<R>(2, k1, a.h, r1, A1, B1, x1); }
                        else { rk_update<R>(3, k0, a.h, r0, A0, B0, x0); rk_update<R>(3, k1, a.h, r1, A1, B1, x1); }
                    }
                    cl.sync();                                   // every CTA is done reading X, Delta and od
                    if (have)
                        for (int c = 0; c < CPS; ++c) {
                            const uint32_t xa = peer_addr(X, (uint32_t)(spin * CPS + c));
                            st_peer(xa + (uint32_t)((j * P + i) * (int)sizeof(cplx<R>)), x0);
                            if (two) st_peer(xa + (uint32_t)((j1 * P + i) * (int)sizeof(cplx<R>)), x1);
                            if (i == j)
                                st_peer(peer_addr(od, (uint32_t)((spin ^ 1) * CPS + c)) + (uint32_t)(i * (int)sizeof(R)), x0.re);
                        }
                    cl.sync();                                   // the next stage input is in place
                }
            }
        }
        if (have) a.state[base + cs(j) + i] = r0;
        if (two) a.state[base + cs(j1) + i] = r1;
        cl.sync();
    }
}

}  // namespace fpsg
