// Exact Hessian sums of the likelihood in one pass over the events.
//
// Compiled by NVRTC for sm_100a on the first request, in a program of its
// own, with "model.cuh" (the model tables) and "model_hess.cuh" (generated:
// the FP64 lineshapes F_t with their first and second theta derivatives).
//
// With z = [Re v, Im v, theta] (HP = 2 M_NA + M_NTH real coordinates, v the
// amplitude couplings) and S_p = sum_a v_a A_{a,p}, an event of weight w adds
// to the Hessian of sum w log f, f = sum_p |S_p|^2,
//   (2 w / f) Re sum_p conj(d_i S_p) d_j S_p - (w / f^2) d_i f d_j f
//     + (2 w / f) Re sum_p conj(S_p) d_i d_j S_p,
// and a phase-space event to that of sum f the first and the third term with
// w / f replaced by 1 (by its weight in the weighted sums). The first two are
// updates of a symmetric HP x HP matrix: per polarisation one of rank two
// with the real and imaginary parts of the HP derivatives d_i S_p, then one
// of rank one. They run on the FP64 tensor cores (mma.sync m8n8k4; tcgen05
// has no FP64 kind), the upper triangle of 8 x 8 blocks in registers: each
// lane forms its own event's derivatives and stores them as columns of a
// [HP][64] slab in shared memory (32 events x re, im), from which the warp
// reads the fragments; both operands of a block product are fragments of the
// same slab, so one 8-byte load per 8 rows and k-step feeds all blocks of
// that row. The third term has few non-zero entries (per derivative entry
// dF_k conj(T), per second derivative v d2F conj(T), T the contraction of the
// angular values with conj(S)): those go to the slab too and each lane sums
// one entry over the 32 events.
//
// What it replaces: forward mode (hessian.cuh) recomputes the lineshapes and
// amplitudes in dual numbers for each of the nparam directions; here they are
// computed once. Per 32 K+K-pi0 events (HP = 23, 3 polarisations) 288 block
// products (336 with the rank-one term), 16 cycles each on a quarter of an
// SM, and ~1600 other FP64 instructions, 2 cycles each: bound by the FP64
// pipe and, at 8 warps per SM (255 registers), by its latency. 11.1M events:
// 30.1 -> 3.8 ms; three chains of rho, 1.11M events: 3.22 -> 0.48 ms (5.4 and
// 0.62 ms with signs and row ends tested in every k-step and four products
// per term and polarisation; 3.95 and 0.51 ms with the rank-one term after the
// polarisations', which keeps its plane sums in registers through them).
//
// Clamps as in the gradient pass: components of w S / f beyond 1e10 count as
// constants (no derivative). Only then are the weights of a polarisation's
// columns masks, and the rank-one term becomes that of two different vectors,
// of which the symmetric part is kept: what a symmetrised Hessian needs. For
// single rows the caller runs forward mode where `clamped` is set.
//
// Each warp strides over 32-event tiles of its CTA's sample; each CTA writes
// one row [HT][8][8] blocks, [M_HLIN] linear sums, sum -w log f; fixed orders
// throughout, so the sums are bit-reproducible.
#pragma once

#include "angular_load.cuh"
#include "device_helpers.cuh"
#include "model.cuh"
#include "model_hess.cuh"

#ifndef CT_HESS_WARPS
#define CT_HESS_WARPS 4
#endif
#ifndef CT_HESS_MINB
#define CT_HESS_MINB 2
#endif
// paired polarisations: table of reals (see hessian.cuh)
#ifndef CT_HESS_PAIRED
#define CT_HESS_PAIRED 0
#endif

#define CT_HP (2 * M_NA + M_NTH)
#define CT_HB ((CT_HP + 7) / 8)
#define CT_HT (CT_HB * (CT_HB + 1) / 2)
#define CT_HROW (CT_HT * 64 + M_HLIN + 1)
// slab row stride in doubles: 64 columns, padded so that 4 consecutive rows
// of a fragment read fall in different banks
#define CT_HRS 68
#define CT_HNPS (CT_HESS_PAIRED ? (M_NPOL + 1) / 2 : M_NPOL)
// a warp's slab: the rows of the matrix (the linear sums' [32][33] use its
// start), then one row of zeros that the lanes of the rows past CT_HP read
#define CT_HROWS (8 * CT_HB * CT_HRS > 32 * 33 ? 8 * CT_HB * CT_HRS : 32 * 33)
#define CT_HSLAB (CT_HROWS + CT_HRS)

struct CtHessConsts {
    double c[M_NHC > 0 ? M_NHC : 1];
    double v[2 * M_NA];
};
__constant__ CtHessConsts hs_k;

struct CtHessSample {
    const void* slamp;     // [M_NPLANE * M_NPOL][ld] angular values, complex, or real when paired
    const double* ev;      // [M_NEV][ld] FP64 frontier values
    const double* w;       // per-event weights or nullptr
    long long n;
    long long ld;
    int kind;   // 0 phase space, 1 data, 2 background
    int group;  // sums it belongs to: 0 phase space, 1 data, 2 background, 3 phase space with its weights
    int cta_begin;
    int cta_count;
};
struct CtHessArgs {
    CtHessSample s[4];
    int nsamp;
    int pad;
    const double* theta;
    const double* v;    // couplings (re, im) x M_NA
    CtHessConsts* img;  // image of hs_k, written by ct_hess_prologue
    double* rows;       // [CTAs][CT_HROW]
    int* clamped;       // set to 1 when an event had clamped components
};

// parameter-only constants (one warp per part, up to 16) and couplings
extern "C" __global__ void __launch_bounds__(512) ct_hess_prologue(CtHessArgs A)
{
    if ((threadIdx.x & 31) == 0)
        for (int q = threadIdx.x >> 5; q < M_NHPRO; q += 16) hs_prologue(q, A.theta, A.img->c);
    for (int i = threadIdx.x; i < 2 * M_NA; i += 512) A.img->v[i] = A.v[i];
    if (threadIdx.x == 0) *A.clamped = 0;
}

__device__ __forceinline__ void ct_dmma(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// One warp's working state for a tile of 32 events (one per lane): the sink
// of hs_columns.
struct CtHessTile {
    double* slab;   // [CT_HSLAB]
    int lane;
    // per event
    double Fr[M_NTERM], Fi[M_NTERM];
    double Wr[M_NDER > 0 ? M_NDER : 1], Wi[M_NDER > 0 ? M_NDER : 1];  // v dF_k
    double2 sl[M_NPLANE * CT_HNPS];
    double cr[M_NPLANE], ci[M_NPLANE];  // sum_p SL_{c,p} conj(u_p), u the clamped w S / f
    double we, alpha, nlog;
    unsigned mask;  // clamped components, 2 p + (0 re, 1 im)
    static_assert(M_NPOL <= 16, "mask of clamped components");
    bool any;       // some lane of the warp clamps
    int kind;
    bool active;
    // per warp
    double lin[(M_HLIN + 31) / 32 > 0 ? (M_HLIN + 31) / 32 : 1];
    double acc[CT_HT][2];
    int row;  // linear sums of this tile written so far

    __device__ __forceinline__ double2 pol(int c, int p) const
    {
        if (!CT_HESS_PAIRED) return sl[c * CT_HNPS + p];
        const int q = M_NPOL - 1 - p;
        if (p < CT_HNPS) return sl[c * CT_HNPS + p];
        const double2 x = sl[c * CT_HNPS + q];
        return make_double2(x.x, -x.y);
    }
    // the polarisation paired with itself: real angular values
    static __device__ __forceinline__ constexpr bool realPol(int p) { return CT_HESS_PAIRED && M_NPOL - 1 - p == p; }
    __device__ __forceinline__ void value(int t, double re, double im)
    {
        Fr[t] = re;
        Fi[t] = im;
    }
    // coherent sums S_p
    __device__ __forceinline__ void coherent(double* Sr, double* Si) const
    {
        double xr[M_NPOL], yi[M_NPOL], yr[M_NPOL], xi[M_NPOL];
#pragma unroll
        for (int p = 0; p < M_NPOL; ++p) xr[p] = yi[p] = yr[p] = xi[p] = 0.0;
#pragma unroll
        for (int t = 0; t < M_NTERM; ++t) {
            const double vr = hs_k.v[2 * term_col(t)], vi = hs_k.v[2 * term_col(t) + 1];
            const double tr = vr * Fr[t] - vi * Fi[t], ti = vr * Fi[t] + vi * Fr[t];
#pragma unroll
            for (int p = 0; p < CT_HNPS; ++p) {
                const double2 x = sl[term_plane(t) * CT_HNPS + p];
                xr[p] += tr * x.x;
                xi[p] += ti * x.x;
                if (!realPol(p)) {
                    yr[p] += tr * x.y;
                    yi[p] += ti * x.y;
                }
            }
        }
        // S_p = sum c (x + iy); paired: S_q = sum c (x - iy) from the same products
#pragma unroll
        for (int p = 0; p < CT_HNPS; ++p) {
            const int q = M_NPOL - 1 - p;
            Sr[p] = realPol(p) ? xr[p] : xr[p] - yi[p];
            Si[p] = realPol(p) ? xi[p] : xi[p] + yr[p];
            if (CT_HESS_PAIRED && q != p) {
                Sr[q] = xr[p] + yi[p];
                Si[q] = xi[p] - yr[p];
            }
        }
    }
    // coherent sums, event weight, contraction of the angular values
    __device__ __forceinline__ void sums()
    {
        double ur[M_NPOL], ui[M_NPOL];
        coherent(ur, ui);
        mask = 0;
        if (kind == 0) {
            alpha = active ? we : 0.0;
#pragma unroll
            for (int p = 0; p < M_NPOL; ++p) {
                ur[p] *= alpha;
                ui[p] *= alpha;
            }
        } else {
            double f = 0.0;
#pragma unroll
            for (int p = 0; p < M_NPOL; ++p) f += ur[p] * ur[p] + ui[p] * ui[p];
            // f == 0: the constant -w log(1e-10), no derivative
            if (active) nlog += f == 0.0 ? -log(1e-10) * we : -log(f) * we;
            alpha = active && f != 0.0 ? we / f : 0.0;
            // (a NaN, 0 times an overflowed w / f, clamps as in forward mode)
#pragma unroll
            for (int p = 0; p < M_NPOL; ++p) {
                ur[p] *= alpha;
                ui[p] *= alpha;
                if (!(fabs(ur[p]) <= 1e10)) mask |= 1u << (2 * p);
                if (!(fabs(ui[p]) <= 1e10)) mask |= 2u << (2 * p);
            }
        }
        any = __any_sync(0xffffffffu, mask != 0);
        if (any) {
#pragma unroll
            for (int p = 0; p < M_NPOL; ++p) {
                ur[p] = fmin(fmax(ur[p], -1e10), 1e10);
                ui[p] = fmin(fmax(ui[p], -1e10), 1e10);
            }
        }
        contract(ur, ui, cr, ci);
        row = 0;
    }
    // (o_r, o_i)_c = sum_p SL_{c,p} conj(u_p)
    __device__ __forceinline__ void contract(const double* ur, const double* ui, double* o_r, double* o_i) const
    {
#pragma unroll
        for (int c = 0; c < M_NPLANE; ++c) {
            double x = 0.0, y = 0.0;
#pragma unroll
            for (int p = 0; p < CT_HNPS; ++p) {
                const int q = M_NPOL - 1 - p;
                const double2 s = sl[c * CT_HNPS + p];
                if (realPol(p)) {
                    x += s.x * ur[p];
                    y -= s.x * ui[p];
                } else if (CT_HESS_PAIRED) {
                    // SL_p conj(u_p) + conj(SL_p) conj(u_q)
                    x += s.x * (ur[p] + ur[q]) + s.y * (ui[p] - ui[q]);
                    y += s.y * (ur[p] - ur[q]) - s.x * (ui[p] + ui[q]);
                } else {
                    x += s.x * ur[p] + s.y * ui[p];
                    y += s.y * ur[p] - s.x * ui[p];
                }
            }
            o_r[c] = x;
            o_i[c] = y;
        }
    }
    // entry `r` of the linear sums: 32 rows of the slab, then a warp-wide flush
    __device__ __forceinline__ void put(int r, double x)
    {
        slab[(r % 32) * 33 + lane] = x;
        if (r % 32 == 31) flush(r / 32, 32);
    }
    __device__ __forceinline__ void flush(int chunk, int rows)
    {
        __syncwarp();
        if (lane < rows) {
            double s = 0.0;
#pragma unroll 8
            for (int e = 0; e < 32; ++e) s += slab[lane * 33 + e];
            lin[chunk] += s;
        }
        __syncwarp();
    }
    __device__ __forceinline__ void der(int k, int t, int r, double re, double im)
    {
        const int a = term_col(t), c = term_plane(t);
        const double vr = hs_k.v[2 * a], vi = hs_k.v[2 * a + 1];
        Wr[k] = vr * re - vi * im;
        Wi[k] = vr * im + vi * re;
        // d2/dRe(v_a)dtheta: 2 Re(dF conj T); d2/dIm(v_a)dtheta: -2 Im(dF conj T)
        put(r, 2.0 * (re * cr[c] - im * ci[c]));
        put(r + 1, -2.0 * (re * ci[c] + im * cr[c]));
    }
    __device__ __forceinline__ void second(int, int t, int r, double re, double im)
    {
        const int a = term_col(t), c = term_plane(t);
        const double vr = hs_k.v[2 * a], vi = hs_k.v[2 * a + 1];
        const double wr = vr * cr[c] - vi * ci[c], wi = vr * ci[c] + vi * cr[c];
        put(r, 2.0 * (re * wr - im * wi));
    }
    // the symmetric update by the slab's KS k-steps of 4 columns (LOGE: log2
    // of the columns per event). SIGN 0: added, 1: subtracted, 2: subtracted
    // for the events of the lanes in `neg`, added for the others
    template <int KS, int LOGE, int SIGN>
    __device__ __forceinline__ void update(unsigned neg)
    {
        __syncwarp();
        const double* base = slab + (lane >> 2) * CT_HRS + (lane & 3);
        const double* last = 8 * (CT_HB - 1) + (lane >> 2) < CT_HP ? base + (CT_HB - 1) * 8 * CT_HRS
                                                                    : slab + CT_HROWS + (lane & 3);
#pragma unroll 4
        for (int s = 0; s < KS; ++s) {
            double b[CT_HB];
#pragma unroll
            for (int I = 0; I < CT_HB; ++I) b[I] = I + 1 < CT_HB ? base[I * 8 * CT_HRS + 4 * s] : last[4 * s];
            const bool minus = SIGN == 2 && ((neg >> ((4 * s + (lane & 3)) >> LOGE)) & 1u);
            int q = 0;
#pragma unroll
            for (int I = 0; I < CT_HB; ++I) {
                const double a = SIGN == 1 || (SIGN == 2 && minus) ? -b[I] : b[I];
#pragma unroll
                for (int J = I; J < CT_HB; ++J) ct_dmma(acc[q++], a, b[J]);
            }
        }
        __syncwarp();
    }
    // rank-one update by the gradient rows of the plane vector (pr, pi):
    // minus its square over w (flip: plus)
    __device__ __forceinline__ void rank1(const double* pr, const double* pi, bool flip)
    {
        const double scale = we != 0.0 ? 1.0 / sqrt(fabs(we)) : 0.0;
        double* o = slab + lane;
#pragma unroll
        for (int a = 0; a < M_NA; ++a) {
            double gr = 0.0, gi = 0.0;
#pragma unroll
            for (int t = 0; t < M_NTERM; ++t)
                if (term_col(t) == a) {
                    const int c = term_plane(t);
                    gr += Fr[t] * pr[c] - Fi[t] * pi[c];
                    gi += Fr[t] * pi[c] + Fi[t] * pr[c];
                }
            o[a * CT_HRS] = scale * gr;
            o[(M_NA + a) * CT_HRS] = -scale * gi;
        }
#pragma unroll
        for (int j = 0; j < M_NTH; ++j) {
            double g = 0.0;
#pragma unroll
            for (int k = 0; k < M_NDER; ++k)
                if (der_th(k) == j) {
                    const int c = term_plane(der_term(k));
                    g += Wr[k] * pr[c] - Wi[k] * pi[c];
                }
            o[(2 * M_NA + j) * CT_HRS] = scale * g;
        }
        // (rows of weight zero are zero, whatever their sign)
        const unsigned neg = __ballot_sync(0xffffffffu, we != 0.0 && (we > 0.0) != flip);
        const unsigned pos = __ballot_sync(0xffffffffu, we != 0.0 && (we > 0.0) == flip);
        if (pos == 0) update<8, 0, 1>(0);
        else update<8, 0, 2>(neg);
    }
    // The plane vectors of a tile with clamps. With y the contraction of all
    // unclamped components w S / f and a that of the components that are not
    // clamped, the rank-one term is minus a y^T / w, symmetrised:
    // (a y^T + y a^T) / 2 = ((a + y)(a + y)^T - (a - y)(a - y)^T) / 4. Both are
    // scaled to the same size first, which leaves their product as it is: y
    // may be 1e10 times a and more, and its square would drown the sums of all
    // other events in rounding. Rare, so the coherent sums are formed again and
    // nothing of this is kept through the derivatives.
    __device__ __forceinline__ void clampedVectors(double* ar, double* ai, double* yr, double* yi) const
    {
        double ur[M_NPOL], ui[M_NPOL];
        coherent(ur, ui);
#pragma unroll
        for (int p = 0; p < M_NPOL; ++p) {
            ur[p] *= alpha;
            ui[p] *= alpha;
        }
        contract(ur, ui, yr, yi);
#pragma unroll
        for (int p = 0; p < M_NPOL; ++p) {
            if ((mask >> (2 * p)) & 1) ur[p] = 0.0;
            if ((mask >> (2 * p)) & 2) ui[p] = 0.0;
        }
        contract(ur, ui, ar, ai);
        double na = 0.0, ny = 0.0;
#pragma unroll
        for (int c = 0; c < M_NPLANE; ++c) {
            na = fmax(na, fmax(fabs(ar[c]), fabs(ai[c])));
            ny = fmax(ny, fmax(fabs(yr[c]), fabs(yi[c])));
        }
        // (all components clamped: a is zero, y possibly infinite)
        const bool none = !(na > 0.0 && ny > 0.0);
        const double sy = none ? 0.0 : sqrt(na / ny), sa = none ? 0.0 : sqrt(ny / na);
#pragma unroll
        for (int c = 0; c < M_NPLANE; ++c) {
            ar[c] *= sa;
            ai[c] *= sa;
            yr[c] = none ? 0.0 : yr[c] * sy;
            yi[c] = none ? 0.0 : yi[c] * sy;
        }
    }
    // (xr, xi) += (fr + i fi) SL_{c,p}
    __device__ __forceinline__ void addProduct(double& xr, double& xi, double fr, double fi, int c, int p) const
    {
        const double2 s = pol(c, p);
        if (realPol(p)) {
            xr += fr * s.x;
            xi += fi * s.x;
        } else {
            xr += fr * s.x - fi * s.y;
            xi += fr * s.y + fi * s.x;
        }
    }
    __device__ __forceinline__ void finish()
    {
        if (M_HLIN % 32) flush(M_HLIN / 32, M_HLIN % 32);
        if (kind != 0) {
            // g = (w / f) grad f, the term -(w / f^2) grad f grad f^T = -g g^T / w
            double pr[M_NPLANE], pi[M_NPLANE];
            if (!any) {
#pragma unroll
                for (int c = 0; c < M_NPLANE; ++c) {
                    pr[c] = 2.0 * cr[c];
                    pi[c] = 2.0 * ci[c];
                }
                rank1(pr, pi, false);
            } else {
                double ar[M_NPLANE], ai[M_NPLANE], yr[M_NPLANE], yi[M_NPLANE];
                clampedVectors(ar, ai, yr, yi);
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int c = 0; c < M_NPLANE; ++c) {
                        pr[c] = ar[c] + (h ? -yr[c] : yr[c]);
                        pi[c] = ai[c] + (h ? -yi[c] : yi[c]);
                    }
                    rank1(pr, pi, h != 0);
                }
            }
        }
        // polarisations: rows sqrt(2 |alpha|) d_i S_p (the factor on the angular values)
        const double sg = sqrt(2.0 * fabs(alpha));
        const unsigned neg = __ballot_sync(0xffffffffu, alpha < 0.0);
#pragma unroll
        for (int c = 0; c < M_NPLANE * CT_HNPS; ++c) {
            sl[c].x *= sg;
            if (!realPol(c % CT_HNPS)) sl[c].y *= sg;
        }
#pragma unroll
        for (int p = 0; p < M_NPOL; ++p) {
            double2* o = reinterpret_cast<double2*>(slab) + lane;
#pragma unroll
            for (int a = 0; a < M_NA; ++a) {
                double xr = 0.0, xi = 0.0;
#pragma unroll
                for (int t = 0; t < M_NTERM; ++t)
                    if (term_col(t) == a) addProduct(xr, xi, Fr[t], Fi[t], term_plane(t), p);
                o[a * (CT_HRS / 2)] = make_double2(xr, xi);
                o[(M_NA + a) * (CT_HRS / 2)] = make_double2(-xi, xr);
            }
#pragma unroll
            for (int j = 0; j < M_NTH; ++j) {
                double xr = 0.0, xi = 0.0;
#pragma unroll
                for (int k = 0; k < M_NDER; ++k)
                    if (der_th(k) == j) addProduct(xr, xi, Wr[k], Wi[k], term_plane(der_term(k)), p);
                o[(2 * M_NA + j) * (CT_HRS / 2)] = make_double2(xr, xi);
            }
            // clamped components drop out
            if (any) {
#pragma unroll 1
                for (int i = 0; i < CT_HP; ++i) {
                    if ((mask >> (2 * p)) & 1) slab[i * CT_HRS + 2 * lane] = 0.0;
                    if ((mask >> (2 * p)) & 2) slab[i * CT_HRS + 2 * lane + 1] = 0.0;
                }
            }
            if (neg == 0) update<16, 1, 0>(0);
            else update<16, 1, 2>(neg);
        }
    }
};

extern "C" __global__ void __launch_bounds__(32 * CT_HESS_WARPS, CT_HESS_MINB) ct_hess_f64(CtHessArgs A)
{
    extern __shared__ __align__(16) double ct_hs[];
    const int cta = (int)blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int si = 0;
#pragma unroll
    for (int k = 1; k < 4; ++k)
        if (k < A.nsamp && cta >= A.s[k].cta_begin) si = k;
    const CtHessSample& S = A.s[si];
    CtHessTile T;
    T.slab = ct_hs + warp * CT_HSLAB;
    for (int i = lane; i < CT_HRS; i += 32) T.slab[CT_HROWS + i] = 0.0;
    T.lane = lane;
    T.kind = S.kind;
    T.nlog = 0.0;
#pragma unroll
    for (int i = 0; i < (M_HLIN + 31) / 32; ++i) T.lin[i] = 0.0;
#pragma unroll
    for (int q = 0; q < CT_HT; ++q) T.acc[q][0] = T.acc[q][1] = 0.0;
    const long long n = S.n, ld = S.ld, ntile = (n + 31) / 32;
    const long long step = (long long)S.cta_count * CT_HESS_WARPS;
    for (long long tile = (long long)(cta - S.cta_begin) * CT_HESS_WARPS + warp; tile < ntile; tile += step) {
        const long long e0 = tile * 32 + lane;
        T.active = e0 < n;
        const long long e = T.active ? e0 : n - 1;  // the tail lanes repeat the last event with weight zero
        double ev[M_NEV > 0 ? M_NEV : 1];
#pragma unroll
        for (int k = 0; k < M_NEV; ++k) ev[k] = __ldg(S.ev + (long long)k * ld + e);
        ct_load_angular<CT_HESS_PAIRED != 0>(S.slamp, ld, e, T.sl);
        T.we = S.w ? __ldg(S.w + e) : 1.0;
        if (!T.active) T.we = 0.0;
        hs_columns(ev, hs_k.c, T);
        T.finish();
        if (T.any && lane == 0) *A.clamped = 1;
    }
    // CTA sums: every warp's sums to its part of shared memory, then added in warp order
    __syncthreads();
    double* part = ct_hs + warp * CT_HROW;
#pragma unroll
    for (int q = 0; q < CT_HT; ++q) {
        part[q * 64 + (lane >> 2) * 8 + 2 * (lane & 3)] = T.acc[q][0];
        part[q * 64 + (lane >> 2) * 8 + 2 * (lane & 3) + 1] = T.acc[q][1];
    }
#pragma unroll
    for (int i = 0; i < (M_HLIN + 31) / 32; ++i)
        if (32 * i + lane < M_HLIN) part[CT_HT * 64 + 32 * i + lane] = T.lin[i];
    double s = T.nlog;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) part[CT_HROW - 1] = s;
    __syncthreads();
    for (int i = threadIdx.x; i < CT_HROW; i += 32 * CT_HESS_WARPS) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < CT_HESS_WARPS; ++w) x += ct_hs[w * CT_HROW + i];
        A.rows[(long long)cta * CT_HROW + i] = x;
    }
}

// Sums of the CTA rows of each group (blockIdx.y; its rows are beg[g], cnt[g]):
// 32 columns per CTA, the rows split over 8 warps and added in a fixed order.
struct CtHessGroups {
    int beg[4], cnt[4];
};
extern "C" __global__ void __launch_bounds__(256) ct_hess_reduce(const double* __restrict__ rows, CtHessGroups G,
                                                                double* __restrict__ sums)
{
    __shared__ double part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = blockIdx.y, col = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (col < CT_HROW) {
#pragma unroll 4
        for (int r = warp; r < G.cnt[g]; r += 8) s += rows[(long long)(G.beg[g] + r) * CT_HROW + col];
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && col < CT_HROW) {
#pragma unroll
        for (int w = 1; w < 8; ++w) s += part[w][lane];
        sums[(long long)g * CT_HROW + col] = s;
    }
}

// Directional sums from the group sums, one CTA of 64 threads per direction u
// (dirs[blockIdx.x], parameter layout): the tangent sums [3][2 + 2 nA + nT]
// of ct_hvp_f64. The CTA after the last direction writes the value sums
// (when vsums is given) of the layout of the gradient pass, of which the
// Hessian's finalize reads the phase-space part and the log-likelihoods.
struct CtHessContractArgs {
    const double* sums;  // [4][CT_HROW]
    const double* dirs;  // [ndir][nparam]
    int ndir, nparam, nc, weighted;  // weighted: group 3 holds the weighted phase-space sums
    const int* chain;
    const double* ratio;
    const double* v;
    double n_phsp, w_phsp, w_data, w_bkg;
    double* tsums;  // [ndir][3][CT_HNACC]
    double* vsums;  // [3][CT_HNACC] + 4, or nullptr
};
#define CT_HNACC (2 + 2 * M_NA + M_NTH)

// component i of (block part) H u
__device__ __forceinline__ double ct_hess_dense(const double* __restrict__ H, const double* u, int i)
{
    double s = 0.0;
    for (int j = 0; j < CT_HP; ++j) {
        const int lo = i < j ? i : j, hi = i < j ? j : i;
        const int I = lo / 8, J = hi / 8;
        const int q = I * CT_HB - I * (I - 1) / 2 + (J - I);
        s += H[q * 64 + (lo % 8) * 8 + hi % 8] * u[j];
    }
    return s;
}
// component i of the linear part
__device__ __forceinline__ double ct_hess_linear(const double* __restrict__ L, const double* u, int i)
{
    double s = 0.0;
    for (int k = 0; k < M_NDER; ++k) {
        const int a = term_col(der_term(k)), j = 2 * M_NA + der_th(k), r = hrow_der(k);
        if (i == a) s += L[r] * u[j];
        if (i == M_NA + a) s += L[r + 1] * u[j];
        if (i == j) s += L[r] * u[a] + L[r + 1] * u[M_NA + a];
    }
    for (int m = 0; m < M_ND2; ++m) {
        const int j0 = 2 * M_NA + d2_th0(m), j1 = 2 * M_NA + d2_th1(m);
        const double x = L[hrow_d2(m)];
        if (i == j0) s += x * u[j1];
        if (j0 != j1 && i == j1) s += x * u[j0];
    }
    return s;
}

extern "C" __global__ void __launch_bounds__(64) ct_hess_contract(CtHessContractArgs A)
{
    __shared__ double u[CT_HP], z0[CT_HP], red[64];
    const int tid = threadIdx.x, d = blockIdx.x;
    const bool value = d == A.ndir;
    for (int i = tid; i < CT_HP; i += 64) {
        const int a = i % M_NA;
        z0[i] = i < 2 * M_NA ? A.v[2 * a + (i >= M_NA)] : 0.0;
        if (value) u[i] = z0[i];
        else {
            const double* dir = A.dirs + (long long)d * A.nparam;
            u[i] = i < 2 * M_NA ? A.ratio[a] * dir[A.chain[a] + (i >= M_NA ? A.nc : 0)] : dir[2 * A.nc + i - 2 * M_NA];
        }
    }
    __syncthreads();
    double* out = value ? A.vsums : A.tsums + (long long)d * 3 * CT_HNACC;
    for (int k = 0; k < 3; ++k) {
        const double* H = A.sums + (long long)k * CT_HROW;
        const double* Hw = A.sums + (long long)(k == 0 && A.weighted ? 3 : k) * CT_HROW;
        double dot = 0.0;
        for (int i = tid; i < CT_HP; i += 64) {
            double hw = ct_hess_dense(i < 2 * M_NA ? Hw : H, u, i);
            // z0 and the block part: sum f = z0 H z0 / 2 and its gradient H z0
            // over phase space; the gradient of sum -w log f is H z0 over the
            // others (H z0 = g - g (g z0) / w with g z0 = 2 w)
            dot += z0[i] * (Hw == H || i >= 2 * M_NA ? hw : ct_hess_dense(H, u, i));
            if (!value) {
                hw += ct_hess_linear((i < 2 * M_NA ? Hw : H) + CT_HT * 64, u, i);
                if (k != 0) hw = -hw;
            }
            const int o = i < M_NA ? 2 + 2 * i : i < 2 * M_NA ? 3 + 2 * (i - M_NA) : 2 + i;
            out[k * CT_HNACC + o] = i < 2 * M_NA ? 0.5 * hw : hw;
        }
        red[tid] = dot;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int i = 0; i < 64; ++i) s += red[i];
            out[k * CT_HNACC + 0] = k == 0 ? 0.0 : value ? H[CT_HROW - 1] : s;
            out[k * CT_HNACC + 1] = k != 0 ? 0.0 : value ? 0.5 * s : s;
        }
        __syncthreads();
    }
    if (value && tid == 0) {
        double* w = A.vsums + 3 * CT_HNACC;
        w[0] = A.n_phsp;
        w[1] = A.w_phsp;
        w[2] = A.w_data;
        w[3] = A.w_bkg;
    }
}
