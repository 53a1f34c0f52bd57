// fpsg_stream_pair.cuh — one RK stage per launch for a Delta with an offset pattern, state
// in HBM: matrices beyond the resident kernels.
//
// k_stream_stage walks Delta's columns by index lists and, when a packed matrix exceeds
// shared memory, gathers its terms from global memory element by element.  Here a thread
// takes slots of two elements, (i, j) and (i, j + 1), lanes consecutive in i, and reads the
// neighbours of the pair at computed distances in the packed columns: every load of a warp is
// one contiguous segment of a column, and the neighbouring columns (off[0] of them on each
// side) stay in L1 while a CTA sweeps its matrix.  What bounds it is HBM traffic: X, rho and
// the two RK accumulators in and out, 19 matrix passes a step.  The lower triangle is read
// as the conjugate of the upper one; only slots within off[0] of the diagonal pay for the
// test.  Sums run in the order of pair_sums_f64 (FP64, the oracle's) or with the diagonal
// term apart (FP32).  16x16 grid, FP32, 512 trajectories, per stage: 713 -> 315 us, 35 % of
// HBM; 15 instructions a term under the masks keep the issue slots at 62 %.  With three offsets
// FP32 spills 280 bytes of stores and 232 of loads per thread at the 64 registers of two CTAs.
#pragma once
#include "fpsg_kernels.cuh"
#include "fpsg_pair.cuh"

namespace fpsg {

constexpr int SP_NT = 512;

template <typename R>
struct StreamPairArgs {
    StreamArgs<R> s;
    Pattern<R> pat;
    const uint32_t* order;    // pair_slot_order
    int nslots;
};

__host__ __device__ __forceinline__ size_t stream_pair_smem(int n, size_t r) 
{
    return sizeof(double) * 64 + align16(r * 2 * (size_t)(n + 1)) + sizeof(uint32_t) * (size_t)(n + 1);
}

template <typename R, int NS>
__global__ void __launch_bounds__(SP_NT, sizeof(R) == 8 ? 1 : 2) k_stream_pair(StreamPairArgs<R> p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const StreamArgs<R>& a = p.s;
    const DevSys<R>& s = a.sys;
    const int n = s.n, ne = s.ne, D = p.pat.off[0], tid = threadIdx.x;
    double* red = reinterpret_cast<double*>(smem);
    R* Dd = reinterpret_cast<R*>(smem + sizeof(double) * 64);
    R* scr = Dd + n + 1;
    uint32_t* mask = reinterpret_cast<uint32_t*>(smem + sizeof(double) * 64 + align16(sizeof(R) * 2 * (size_t)(n + 1)));
    for (int j = tid; j <= n; j += SP_NT) mask[j] = j < n ? p.pat.mask[j] : 0u;
    for (int m = blockIdx.x; m < 2 * a.B; m += gridDim.x) {
        const cplx<R>* X = a.Xc + (size_t)m * ne;
        const cplx<R>* xo = a.Xc + (size_t)(m ^ 1) * ne;
        __syncthreads();
        if (s.ud == nullptr) {
            for (int j = tid; j < n; j += SP_NT) Dd[j] = delta_diag<R>(s, j, X, xo, a.pulse);
        } else {
            // dense Coulomb rows: ascending k per site, U and V sums on separate threads
            for (int q = tid; q < 2 * n; q += SP_NT) {
                const bool vt = q >= n;
                const int j = vt ? q - n : q;
                const cplx<R>* d = vt ? X : xo;
                const R* c = (vt ? s.vd : s.ud) + j;
                R u = R(0);
                if (!vt || s.coul == 2)
#pragma unroll 8
                    for (int k = 0; k < n; ++k) u = fmaR<R>(c[(size_t)k * n], addR<R>(d[cs(k) + k].re, s.shift), u);
                (vt ? scr : Dd)[j] = u;
            }
            __syncthreads();
            for (int j = tid; j < n; j += SP_NT) {
                R d = addR<R>(s.tdiag[j], Dd[j]);
                if (s.coul == 2) d = addR<R>(d, scr[j]);
                if (s.has_ext) d = addR<R>(d, s.ediag[j]);
                if (s.n_bins > 0) d = addR<R>(d, mulR<R>(a.pulse, s.proj[j]));
                Dd[j] = d;
            }
        }
        if (tid == 0) Dd[n] = R(0);
        if (a.record) {
            for (int j = tid; j < n; j += SP_NT) {
                const double d = (double)X[cs(j) + j].re;
                if (!isfinite(d)) atomicOr(a.err, 1u);
                a.diagbuf[(size_t)m * n + j] = d;
            }
            double e[4] = {0.0, 0.0, 0.0, 0.0};
            energy_partials<R>(s, X, xo, m & 1, a.do_e1, a.do_e2, tid, SP_NT, e);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double v = warp_sum(e[c]);
                if ((tid & 31) == 0) red[(tid >> 5) * 4 + c] = v;
            }
            __syncthreads();
            if (tid < 4) {
                double v = 0.0;
                for (int q = 0; q < SP_NT / 32; ++q) v += red[q * 4 + tid];
                a.ebuf[(size_t)m * 4 + tid] = v;
            }
            if (a.whole)
                for (int q = tid; q < ne; q += SP_NT) {
                    atomicAdd(&a.whole[(size_t)(m & 1) * ne + q].x, (double)X[q].re);
                    atomicAdd(&a.whole[(size_t)(m & 1) * ne + q].y, (double)X[q].im);
                }
        }
        __syncthreads();
        for (int f = tid; f < p.nslots; f += SP_NT) {
            const uint32_t code = p.order[f];
            if (code == ~0u) continue;
            const int i = (int)(code & 0xffffu), j = (int)((code >> 16) & 0x7fffu);
            const bool one = (code & PAIR_NONE) != 0;
            const uint32_t mi = mask[i], m0 = mask[j], m1 = one ? 0u : mask[j + 1];
            // every term's load first, at the slot's own element where there is no such neighbour
            // (loads under their masks went out one after the other)
            cplx<R> o0, o1, xa[2][NS][2], xb[2][NS][2];   // [element][offset][below, above]: columns, rows
            auto load = [&](auto at) {
                o0 = at(0, 0, true);
                o1 = at(0, 1, !one);
#pragma unroll
                for (int q = 0; q < NS; ++q) {
                    const int o = p.pat.off[q];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int sg = u ? o : -o;
                        const bool row = (mi >> (2 * q + u)) & 1u;
                        xa[0][q][u] = q == NS - 1 && u == 1 ? o1 : at(0, sg, (m0 >> (2 * q + u)) & 1u);
                        xa[1][q][u] = q == NS - 1 && u == 0 ? o0 : at(0, 1 + sg, (m1 >> (2 * q + u)) & 1u);
                        xb[0][q][u] = at(sg, 0, row);
                        xb[1][q][u] = at(sg, 1, row && !one);
                    }
                }
                if (one && ((m0 >> (2 * NS - 1)) & 1u)) xa[0][NS - 1][1] = at(0, 1, true);
            };
            // (dr, dc): row i + dr, column j + dc
            const cplx<R>* xp = X + cs(j) + i;
            if (__any_sync(__activemask(), j - i <= D + 1)) {     // some neighbour may lie in the lower triangle
                load([&](int dr, int dc, bool ok) -> cplx<R> {
                    const int r = i + dr, c = j + dc;
                    const int hi = ok ? max(r, c) : j, lo = ok ? min(r, c) : i;
                    cplx<R> v = X[cs(hi) + lo];
                    if (r > c) v.im = -v.im;
                    return v;
                });
            } else {
                load([&](int dr, int dc, bool ok) -> cplx<R> {
                    const int d = dc * j + ((dc * (dc + 1)) >> 1) + dr;      // cs(j + dc) - cs(j) + dr
                    return xp[ok ? d : 0];
                });
            }
            const size_t g0 = (size_t)m * ne + cs(j) + i, g1 = g0 + j + 1;
            const cplx<R> z = {R(0), R(0)};
            cplx<R> r0 = o0, r1 = o1, A0 = z, A1 = z, B0 = z, B1 = z;
            if (a.stage != 0) { r0 = a.rho[g0]; if (!one) r1 = a.rho[g1]; }
            if (a.stage == 1 || a.stage == 2) { A0 = a.A[g0]; if (!one) A1 = a.A[g1]; }
            if (a.stage >= 2) { B0 = a.Bc[g0]; if (!one) B1 = a.Bc[g1]; }
            const R di = Dd[i], d0 = Dd[j], d1 = Dd[j + 1];
            R a0r = R(0), a0i = R(0), a1r = R(0), a1i = R(0), c0r = R(0), c0i = R(0), c1r = R(0), c1i = R(0);
            auto add = [&](R& re, R& im, const cplx<R>& x, bool ok) {
                if (ok) { re = fmaR<R>(x.re, p.pat.w, re); im = fmaR<R>(x.im, p.pat.w, im); }
            };
            auto side = [&](int u) {
#pragma unroll
                for (int t = 0; t < NS; ++t) {
                    const int q = u ? NS - 1 - t : t;             // ascending k
                    const bool row = (mi >> (2 * q + u)) & 1u;
                    add(a0r, a0i, xa[0][q][u], (m0 >> (2 * q + u)) & 1u);
                    add(a1r, a1i, xa[1][q][u], (m1 >> (2 * q + u)) & 1u);
                    add(c0r, c0i, xb[0][q][u], row);
                    add(c1r, c1i, xb[1][q][u], row);
                }
            };
            side(0);
            if constexpr (!std::is_same<R, float>::value) {
                a0r = fmaR<R>(o0.re, d0, a0r); a0i = fmaR<R>(o0.im, d0, a0i);
                c0r = fmaR<R>(o0.re, di, c0r); c0i = fmaR<R>(o0.im, di, c0i);
                a1r = fmaR<R>(o1.re, d1, a1r); a1i = fmaR<R>(o1.im, d1, a1i);
                c1r = fmaR<R>(o1.re, di, c1r); c1i = fmaR<R>(o1.im, di, c1i);
            }
            side(1);
            if constexpr (std::is_same<R, float>::value) {
                a0r = fmaR<R>(o0.re, d0 - di, a0r); a0i = fmaR<R>(o0.im, d0 - di, a0i);
                a1r = fmaR<R>(o1.re, d1 - di, a1r); a1i = fmaR<R>(o1.im, d1 - di, a1i);
            }
            cplx<R> x0, x1;
            rk_update<R>(a.stage, cplx<R>{subR<R>(a0i, c0i), -subR<R>(a0r, c0r)}, a.h, r0, A0, B0, x0);
            rk_update<R>(a.stage, cplx<R>{subR<R>(a1i, c1i), -subR<R>(a1r, c1r)}, a.h, r1, A1, B1, x1);
            if (a.stage <= 1) { a.A[g0] = A0; if (!one) a.A[g1] = A1; }
            if (a.stage == 1 || a.stage == 2) { a.Bc[g0] = B0; if (!one) a.Bc[g1] = B1; }
            if (a.stage < 3) { a.Xn[g0] = x0; if (!one) a.Xn[g1] = x1; }
            else { a.rho[g0] = r0; if (!one) a.rho[g1] = r1; }
        }
    }
}

}  // namespace fpsg
