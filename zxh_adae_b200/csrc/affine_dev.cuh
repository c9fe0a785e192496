// affine_dev.cuh -- device side of the affine tile pass: shared by its own kernel (affine.cu,
// which describes it) and the persistent batch kernel (batch.cu).
#pragma once

#include "affine.h"
#include "chain.cuh"
#include "core.h"
#include "dev.cuh"

#include <cuda_runtime.h>

#include <type_traits>

namespace zxh {
namespace adev {

constexpr int kNR = 16;   // amplitudes per thread
constexpr int kRun = 1 << kAffRun;
constexpr int kSums = 11;  // w summed over a thread's registers: all, 4 bits, 6 pairs of bits

template <typename E, bool ADJ>
struct AffSmem {
    using RT = typename ET<E>::R;
    static constexpr int NW = ADJ ? 1 : 2;  // windows
    // The windows' entries: in shared memory, but for complex128 forward passes, where L1 serves
    // the space better (24-qubit ansatz 2.86 -> 2.64 ms; complex64 1.32 -> 1.36).
    static constexpr bool ENT = ADJ || sizeof(E) == 8;
    E slab[ADJ ? 2 : 1][1 << kAffBits];      // adjoint passes: also the sums and marginals of w
    E exp[1 << kExpTableBits];
    RT u[kAffBits][2][8];  // [1]: the |1> member first
    RT rot[kAffBits];
    double gscale[kAffBits];
    uint32_t sel[kAffBits], gen[kAffBits];
    uint64_t lw[kRun];
    uint32_t alpha[kAffMaxSel], basis[kAffBits];
    AffWinDev win[NW];
    AffEntryDev ent[ENT ? NW : 1][ENT ? kAffMaxEntries : 1];
    int64_t K[NW][kRun], w[NW][kRun][kAffHigh], q[NW][kRun][kAffPairs];
    AffTermDev term[ADJ ? kAffMaxTerms : 1];
    uint8_t plist[kAffPairs];
    double tacc[ADJ ? kAffMaxTerms : 1];
    double gacc[ADJ ? kAffBits : 1][ADJ ? kThreads : 1];
};

// SWZ: the exchanges of layout C, whose half warps differ in coordinates 4..7; between A and B
// (coordinates 0..3) the plain index serves, with every register at a constant offset.
template <bool SWZ>
__host__ __device__ constexpr uint32_t slot_of(uint32_t i) { return SWZ ? i ^ ((i >> 4) & 15u) : i; }

// Registers j of layout L (0 A, 1 B, 2 C) in tile index bits.
template <int L>
__host__ __device__ constexpr uint32_t reg_bits(int j) { return L == 0 ? uint32_t(j) << 4 : L == 1 ? uint32_t(j) << 8 : uint32_t(j); }
template <int L>
__device__ __forceinline__ uint32_t fixed_bits(uint32_t lane, uint32_t warp)
{
    if constexpr (L == 0) return (lane & 15u) | ((lane >> 4) << 8) | (warp << 9);
    if constexpr (L == 1) return lane | (warp << 5);
    return (lane << 4) | (warp << 9);
}

template <int LA, int LB, int NS, typename E>
__device__ __forceinline__ void exchange(E (&x)[kNR], E (&y)[kNR], E (*slab)[1 << kAffBits], uint32_t lane, uint32_t warp)
{
    constexpr bool SWZ = LA == 2 || LB == 2;
    const uint32_t a = slot_of<SWZ>(fixed_bits<LA>(lane, warp)), b = slot_of<SWZ>(fixed_bits<LB>(lane, warp));
    __syncthreads();  // the slab's previous reads are done
#pragma unroll
    for (int j = 0; j < kNR; j++) {
        const uint32_t s = SWZ ? a ^ slot_of<SWZ>(reg_bits<LA>(j)) : a + reg_bits<LA>(j);
        slab[0][s] = x[j];
        if constexpr (NS == 2) slab[1][s] = y[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kNR; j++) {
        const uint32_t s = SWZ ? b ^ slot_of<SWZ>(reg_bits<LB>(j)) : b + reg_bits<LB>(j);
        x[j] = slab[0][s];
        if constexpr (NS == 2) y[j] = slab[1][s];
    }
}

template <typename E, typename RT>
__device__ __forceinline__ E cmad2(RT ar, RT ai, E a, RT br, RT bi, E b)  // a-coefficient * a + b-coefficient * b
{
    E o;
    o.x = ar * a.x - ai * a.y + br * b.x - bi * b.y;
    o.y = ar * a.y + ai * a.x + br * b.y + bi * b.x;
    return o;
}

// a * b + c by components (the real parts of conj(a) b summed over both).
__device__ __forceinline__ float2 dot2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ double2 dot2(double2 a, double2 b, double2 c)
{
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}

// The gate on register bit RR, m its matrix in the thread's orientation; adjoint passes
// first add the gradient's share (FP32 over 8 pairs for complex64) to acc.
template <int RR, bool ADJ, bool REAL, typename E, typename RT>
__device__ __forceinline__ void gate(E (&x)[kNR], E (&y)[kNR], const RT *m, bool flip, uint32_t gen, double *acc)
{
    [[maybe_unused]] E p0 = {0, 0}, p1 = {0, 0};
    const RT m0 = m[0], m2 = m[2], m4 = m[4], m6 = m[6];
    const RT m1 = REAL ? RT(0) : m[1], m3 = REAL ? RT(0) : m[3], m5 = REAL ? RT(0) : m[5], m7 = REAL ? RT(0) : m[7];
#pragma unroll
    for (int j = 0; j < kNR; j++) {
        if ((j >> RR) & 1) continue;
        constexpr int B = 1 << RR;
        const E lo = x[j], hi = x[j | B];
        if constexpr (ADJ) {
            const E llo = y[j], lhi = y[j | B];
            if (gen == 1) {  // Im<l|Y|p> = Re(conj(l1) p0) - Re(conj(l0) p1)
                p0 = dot2(lhi, lo, p0);
                p1 = dot2(llo, hi, p1);
            } else if (gen == 2) {  // Im<l|X|p> = Im(conj(l0) p1 + conj(l1) p0)
                p0.x += llo.x * hi.y - llo.y * hi.x;
                p0.y += lhi.x * lo.y - lhi.y * lo.x;
            }
            if constexpr (REAL) {
                y[j] = rmad2(m0, llo, m2, lhi);
                y[j | B] = rmad2(m4, llo, m6, lhi);
            } else {
                y[j] = cmad2(m0, m1, llo, m2, m3, lhi);
                y[j | B] = cmad2(m4, m5, llo, m6, m7, lhi);
            }
        }
        if constexpr (REAL) {
            x[j] = rmad2(m0, lo, m2, hi);
            x[j | B] = rmad2(m4, lo, m6, hi);
        } else {
            x[j] = cmad2(m0, m1, lo, m2, m3, hi);
            x[j | B] = cmad2(m4, m5, lo, m6, m7, hi);
        }
    }
    if constexpr (ADJ) {
        if (gen == 1) {
            const double part = (double(p0.x) - double(p1.x)) + (double(p0.y) - double(p1.y));
            *acc += flip ? -part : part;
        } else if (gen == 2) {
            *acc += double(p0.x) + double(p0.y);
        }
    }
}

__device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ double2 neg(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ float2 axpy(float c, float2 a, float2 b) { return __ffma2_rn(make_float2(c, c), a, b); }
__device__ __forceinline__ double2 axpy(double c, double2 a, double2 b)
{
    return make_double2(fma(c, a.x, b.x), fma(c, a.y, b.y));
}
__device__ __forceinline__ float2 scaled(float c, float2 a) { return __fmul2_rn(make_float2(c, c), a); }
__device__ __forceinline__ double2 scaled(double c, double2 a) { return make_double2(c * a.x, c * a.y); }

// One half of a factored gate on a state: lo' = a lo + p hi, hi' = q lo + b hi with
//   rotation   (rot = s / c)  lo - r hi, hi + r lo     (rot = c / s)  r lo - hi, lo + r hi
//   reflection (rot = s / c)  lo + r hi, r lo - hi     (rot = c / s)  r lo + hi, lo - r hi
template <int RR, bool MU, bool REFL, typename E, typename RT>
__device__ __forceinline__ void factored(E (&x)[kNR], RT r)
{
    constexpr int B = 1 << RR;
    const RT nr = -r;
#pragma unroll
    for (int j = 0; j < kNR; j++) {
        if ((j >> RR) & 1) continue;
        const E lo = x[j], hi = x[j | B];
        if constexpr (!MU && !REFL) {
            x[j] = axpy(nr, hi, lo);
            x[j | B] = axpy(r, lo, hi);
        } else if constexpr (!REFL) {
            x[j] = axpy(r, lo, neg(hi));
            x[j | B] = axpy(r, hi, lo);
        } else if constexpr (!MU) {
            x[j] = axpy(r, hi, lo);
            x[j | B] = axpy(r, lo, neg(hi));
        } else {
            x[j] = axpy(r, lo, hi);
            x[j | B] = axpy(nr, hi, lo);
        }
    }
}

// A rotation or reflection with one coefficient factored out: half the multiply-adds of
// gate(), and one rounding less. r: its coefficient, negated where the thread's pairs start
// at the |1> member (flip). One branch per form around whole loops: inside them the compiler
// computes every form.
template <int RR, bool ADJ, typename E, typename RT>
__device__ __forceinline__ void factored_gate(E (&x)[kNR], E (&y)[kNR], RT r, bool mu, bool refl, bool flip, uint32_t gen,
                                              double gscale, double *acc)
{
    constexpr int B = 1 << RR;
    if constexpr (ADJ) {
        if (gen) {
            E p0 = {0, 0}, p1 = {0, 0};
#pragma unroll
            for (int j = 0; j < kNR; j++) {
                if ((j >> RR) & 1) continue;
                p0 = dot2(y[j | B], x[j], p0);
                p1 = dot2(y[j], x[j | B], p1);
            }
            const double part = (double(p0.x) - double(p1.x)) + (double(p0.y) - double(p1.y));
            *acc += gscale * (flip ? -part : part);
        }
    }
    auto both = [&](auto m, auto f) {
        factored<RR, decltype(m)::value, decltype(f)::value>(x, r);
        if constexpr (ADJ) factored<RR, decltype(m)::value, decltype(f)::value>(y, r);
    };
    using T = std::true_type;
    using F = std::false_type;
    if (!refl) {
        if (mu) both(T(), F());
        else both(F(), F());
    } else {
        if (mu) both(T(), T());
        else both(F(), T());
    }
}

// The gates on coordinates K0 .. K0 + 3, the layout's registers; c: the selector bits of
// the thread (of the tile, in layout C).
template <int K0, bool ADJ, int FORM, typename E, typename SM>
__device__ __forceinline__ void gates(E (&x)[kNR], E (&y)[kNR], uint32_t mask, uint32_t mu, uint32_t refl, uint64_t c, SM &sm,
                                      uint32_t tid)
{
    auto one = [&](auto rr) {
        constexpr int RR = decltype(rr)::value, k = K0 + RR;
        if (!((mask >> k) & 1u)) return;
        const bool flip = (uint32_t(c) >> sm.sel[k]) & 1u;  // the gates' selectors are the first ones
        double *acc = ADJ ? &sm.gacc[ADJ ? k : 0][ADJ ? tid : 0] : nullptr;
        if constexpr (FORM == 2) {
            const auto r = sm.rot[k];
            factored_gate<RR, ADJ>(x, y, flip ? -r : r, (mu >> k) & 1u, (refl >> k) & 1u, flip, sm.gen[k], sm.gscale[k], acc);
        } else {
            gate<RR, ADJ, FORM == 1>(x, y, sm.u[k][flip], flip, sm.gen[k], acc);
        }
    };
    one(std::integral_constant<int, 0>());
    one(std::integral_constant<int, 1>());
    one(std::integral_constant<int, 2>());
    one(std::integral_constant<int, 3>());
}

// Window d's polynomial at run position l, by the 16 threads part = 0..15 of that position:
// all take shares of the entries without a coordinate, thread k < 8 those of coordinate k.
template <typename SM>
__device__ __forceinline__ void window_eval(SM &sm, const AffEntryDev *ent, const AffWinDev &wd, int d, uint64_t c,
                                            uint32_t part, uint32_t l)
{
    int64_t K = 0;
    for (uint32_t e = part; e < wd.n0; e += 16u) {
        const AffEntryDev t = ent[e];
        const bool on = ((c >> t.s0) & 1) && (t.s1 == 0xff || ((c >> t.s1) & 1));
        if (on) K += t.coef;
    }
    if (part < uint32_t(kAffHigh)) {
        int64_t w = 0;
        for (uint32_t e = wd.ck[part]; e < wd.ck[part + 1]; e++) {
            const AffEntryDev t = ent[e];
            const bool f0 = (c >> t.s0) & 1, f1 = t.s1 != 0xff && ((c >> t.s1) & 1);
            const int64_t slope = f0 ? -t.coef : t.coef;  // S = f + y (1 - 2 f)
            if (t.kind == 3) {
                if (f0 && f1) K += t.coef;
                if (f1) w += slope;
                const int64_t q = f0 != f1 ? -t.coef : t.coef;
                sm.q[d][l][t.pair] = t.first ? q : sm.q[d][l][t.pair] + q;
            } else if (t.kind == 4) {
                if (f1) w += slope;
            } else if (t.kind == 1 || (t.kind == 2 ? f1 : f0 == f1)) {
                if (f0) K += t.coef;
                w += slope;
            }
        }
        sm.w[d][l][part] = w;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) K += __shfl_xor_sync(0xffffffffu, K, o);
    if (part == 0) sm.K[d][l] = K;
}

template <typename E>
struct Turn;  // turns of a phase in the state's precision
template <>
struct Turn<float2> {
    using T = uint32_t;
    static __device__ __forceinline__ T of(int64_t t) { return turns32(t); }
    static __device__ __forceinline__ float2 factor(const float2 *tab, T t) { return phase_factor32(tab, t); }
};
template <>
struct Turn<double2> {
    using T = int64_t;
    static __device__ __forceinline__ T of(int64_t t) { return t; }
    static __device__ __forceinline__ double2 factor(const double2 *tab, T t) { return phase_factor(tab, t); }
};

// Window d applied in layout L (A: registers are high coordinates 0..3 and the thread
// fixes 4..7; B: the other way round).
template <int L, bool ADJ, typename E, typename SM>
__device__ __forceinline__ void window_apply(E (&x)[kNR], E (&y)[kNR], SM &sm, uint32_t pairs, int d, uint32_t lane,
                                             uint32_t warp)
{
    constexpr int RK = L == 0 ? 0 : 4, FK = 4 - RK;  // first register / fixed high coordinate
    const uint32_t l = lane & 15u, fix = (lane >> 4) | (warp << 1);
    int64_t a = sm.K[d][l], w[4], q[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if ((fix >> i) & 1u) a += sm.w[d][l][FK + i];
        w[i] = sm.w[d][l][RK + i];
    }
    if (pairs) {
#pragma unroll
        for (int i = 0; i < kAffHigh; i++)
#pragma unroll
            for (int j = i + 1; j < kAffHigh; j++) {
                if (!((pairs >> aff_pair(i, j)) & 1u)) continue;
                const int64_t v = sm.q[d][l][aff_pair(i, j)];
                const bool ri = i >= RK && i < RK + 4, rj = j >= RK && j < RK + 4;
                if (ri && rj) {
                    constexpr int base[4] = {0, 3, 5, 6};
                    q[base[i & 3] + (j & 3) - (i & 3) - 1] = v;
                } else if (!ri && !rj) {
                    if ((fix >> (i & 3)) & (fix >> (j & 3)) & 1u) a += v;
                } else if ((fix >> ((ri ? j : i) & 3)) & 1u) {
                    w[(ri ? i : j) & 3] += v;
                }
            }
    }
    using TT = typename Turn<E>::T;
    const TT ta = Turn<E>::of(a);
    TT tw[4], tq[6];
#pragma unroll
    for (int i = 0; i < 4; i++) tw[i] = Turn<E>::of(w[i]);
#pragma unroll
    for (int i = 0; i < 6; i++) tq[i] = Turn<E>::of(q[i]);
#pragma unroll
    for (int j = 0; j < kNR; j++) {
        TT t = ta;
#pragma unroll
        for (int b = 0; b < 4; b++)
            if ((j >> b) & 1) t += tw[b];
        int n = 0;
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
            for (int e = b + 1; e < 4; e++, n++)
                if (((j >> b) & 1) && ((j >> e) & 1)) t += tq[n];
        const E ph = Turn<E>::factor(sm.exp, t);
        x[j] = cmul(x[j], ph);
        if constexpr (ADJ) y[j] = cmul(y[j], ph);
    }
}

// The window's gradients, in layout A before its phases are undone: per run position the
// sum of w and its marginals over the high coordinates and their pairs, then each term's
// sum_r w (S ? m1 : m0) from them. P: the tile's selector bits.
template <typename E, typename SM>
__device__ __forceinline__ void window_grad(const E (&x)[kNR], const E (&y)[kNR], SM &sm, const AffWinDev &wd, uint64_t P,
                                            uint32_t tid)
{
    double *V = reinterpret_cast<double *>(&sm.slab[0][0]);  // [kSums][16 fixed][16 run]
    double *M = V + kSums * kThreads;                         // [1 + 8 + pairs][16 run]
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const uint32_t pairs = wd.pairs;
    {
        double v[kSums];
#pragma unroll
        for (int i = 0; i < kSums; i++) v[i] = 0.0;
#pragma unroll
        for (int j = 0; j < kNR; j++) {
            const double w = double(y[j].x * x[j].y - y[j].y * x[j].x);  // Im(conj(lambda) psi)
            v[0] += w;
            int n = 5;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                if ((j >> b) & 1) v[1 + b] += w;
#pragma unroll
                for (int e = b + 1; e < 4; e++, n++)
                    if (((j >> b) & 1) && ((j >> e) & 1)) v[n] += w;
            }
        }
        const uint32_t at = (((lane >> 4) | (warp << 1)) << 4) | (lane & 15u);
#pragma unroll
        for (int i = 0; i < kSums; i++)
            if (i < 5 || pairs) V[i * kThreads + at] = v[i];
    }
    __syncthreads();
    const uint32_t l = tid & 15u, part = tid >> 4;
    const uint32_t rows = 9u + uint32_t(__popc(pairs));
    for (uint32_t r = part; r < rows; r += 16u) {
        uint32_t src = 0, need = 0;  // row of V, fixed bits that must be set
        if (r >= 1 && r < 9) {
            if (r < 5) src = r;
            else need = 1u << (r - 5);
        } else if (r >= 9) {
            const uint32_t p = sm.plist[r - 9];
            const uint32_t i = p & 15u, j = p >> 4;
            if (j < 4) src = 5u + (i == 0 ? j - 1 : i == 1 ? j + 1 : 5u);  // (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
            else if (i < 4) src = 1u + i, need = 1u << (j - 4);
            else need = (1u << (i - 4)) | (1u << (j - 4));
        }
        double s = 0.0;
#pragma unroll
        for (uint32_t f = 0; f < 16; f++)
            if ((f & need) == need) s += V[src * kThreads + (f << 4) + l];
        M[r * kRun + l] = s;
    }
    __syncthreads();
    const uint64_t c = P ^ sm.lw[l];
    const double W = M[l];
    for (uint32_t t0 = 0; t0 < wd.nterms; t0 += 16u) {
        const uint32_t t = t0 + part;
        const bool live = t < wd.nterms;
        const AffTermDev tm = sm.term[live ? t : 0];
        const bool f0 = (c >> tm.s0) & 1, two = tm.s1 != 0xff, f1 = two && ((c >> tm.s1) & 1);
        double s;
        if (tm.k0 == 0xff) {
            s = f0 && (!two || f1) ? W : 0.0;
        } else {
            const double M0 = M[(1u + tm.k0) * kRun + l], S0 = f0 ? W - M0 : M0;
            if (!two) s = S0;
            else if (tm.k1 == 0xff) s = f1 ? S0 : 0.0;
            else if (tm.k1 == tm.k0) s = f0 == f1 ? S0 : 0.0;
            else {
                const double M1 = M[(1u + tm.k1) * kRun + l], M01 = M[(9u + tm.pair) * kRun + l];
                s = f0 ? (f1 ? W - M0 - M1 + M01 : M1 - M01) : (f1 ? M0 - M01 : M01);
            }
        }
        const double g0 = tm.gk == 1 ? 1.0 : 0.0, g1 = tm.gk == 1 ? -1.0 : -2.0;
        double g = live && tm.gk ? g0 * W + (g1 - g0) * s : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
        if (live && l == 0) sm.tacc[t] += g;
    }
}

// The pass on the calling CTA of 256 threads over tiles first, first + step, ... below end;
// a launch
// that may have started before the work it follows has ended waits for it here (chain.cuh):
// nothing but the program is read before that.
template <typename E, bool ADJ, int FORM>
__device__ __forceinline__ void affine_body(AffSmem<E, ADJ> &sm, const uint8_t *__restrict__ blob, uint64_t poff,
                                            uint64_t toff, E *psi, const E *src, E *lam, double *grads, uint32_t first,
                                            uint32_t step, uint32_t end)
{
    using SM = AffSmem<E, ADJ>;
    using RT = typename ET<E>::R;
    const AffDev &p = *reinterpret_cast<const AffDev *>(blob + poff);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t mask = p.gates, mu = p.mu, refl = p.refl, nsel = p.nsel;
    const uint64_t neg_high = p.neg_high, neg_low = p.neg_low;
    const RT scale = RT(p.scale);
    const AffWinDev &w0 = sm.win[0], &w1 = sm.win[SM::NW - 1];
    const bool win0 = p.win[0].nterms != 0, win1 = !ADJ && p.win[1].nterms != 0;

    // tables
    __syncthreads();  // they may still be read by an earlier call
    if (tid < SM::NW) sm.win[tid] = p.win[tid];
    __syncthreads();
    if (win0 || win1) {
        const E *tab = reinterpret_cast<const E *>(blob + toff);
        for (uint32_t i = tid; i < (1u << kExpTableBits); i += kThreads) sm.exp[i] = tab[i];
        if constexpr (SM::ENT)
            for (int d = 0; d < SM::NW; d++) {
                const AffEntryDev *e = reinterpret_cast<const AffEntryDev *>(blob + sm.win[d].off_entries);
                for (uint32_t i = tid; i < sm.win[d].ck[kAffHigh]; i += kThreads) sm.ent[d][i] = e[i];
            }
    }
    if (tid < kAffBits) {
        const AffGateDev &g = p.gate[tid];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            sm.u[tid][0][i] = RT(g.u[i]);
            sm.u[tid][1][i] = RT(g.u[i ^ 6]);  // [[u11, u10], [u01, u00]]
        }
        sm.rot[tid] = RT(g.rot);
        sm.gscale[tid] = g.gscale;
        sm.sel[tid] = g.sel;
        sm.gen[tid] = g.gen;
        sm.basis[tid] = uint32_t(p.basis[tid]);
    }
    if (tid >= 32 && tid < 32 + kAffMaxSel) sm.alpha[tid - 32] = uint32_t(p.alpha[tid - 32]);
    if (tid >= 96 && tid < 96 + kRun) sm.lw[tid - 96] = p.lw[tid - 96];
    if constexpr (ADJ) {
        const AffTermDev *t = reinterpret_cast<const AffTermDev *>(blob + w0.off_terms);
        for (uint32_t i = tid; i < w0.nterms; i += kThreads) {
            sm.term[i] = t[i];
            sm.tacc[i] = 0.0;
        }
#pragma unroll
        for (int k = 0; k < kAffBits; k++) sm.gacc[k][tid] = 0.0;
        if (tid == 128) {
            int n = 0;
            for (int i = 0; i < kAffHigh; i++)
                for (int j = i + 1; j < kAffHigh; j++)
                    if ((w0.pairs >> aff_pair(i, j)) & 1u) sm.plist[n++] = uint8_t(i | (j << 4));
        }
    }
    __syncthreads();

    // the thread's part of the address in layouts A and B
    uint32_t ra = 0, rb = 0;
#pragma unroll
    for (int b = 0; b < 5; b++)
        if ((lane >> b) & 1u) {
            ra ^= sm.basis[b < 4 ? b : 8];
            rb ^= sm.basis[b];
        }
#pragma unroll
    for (int b = 0; b < 3; b++)
        if ((warp >> b) & 1u) {
            ra ^= sm.basis[9 + b];
            rb ^= sm.basis[5 + b];
        }
    const uint32_t trl = uint32_t(p.tr[lane]);  // at most 20 tile bits
    auto entries = [&](int d) {
        return SM::ENT ? sm.ent[SM::ENT ? d : 0] : reinterpret_cast<const AffEntryDev *>(blob + sm.win[d].off_entries);
    };
    const AffEntryDev *ent0 = entries(0);
    [[maybe_unused]] const AffEntryDev *ent1 = entries(SM::NW - 1);
    const bool need_c = (mask & 0x00fu) != 0, need_b = need_c || (mask & 0xf00u) != 0 || win1;
    const uint64_t lw = sm.lw[lane & 15u], lw0 = sm.lw[0], lwe = sm.lw[tid >> 4];

    auto tile_base = [&](uint32_t t) { return __reduce_xor_sync(0xffffffffu, ((t >> lane) & 1u) ? trl : 0u); };
    // the run of 16 amplitudes this thread asks L2 for, one tile ahead
    uint32_t rp = 0;
#pragma unroll
    for (int b = 0; b < kAffHigh; b++)
        if ((tid >> b) & 1u) rp ^= sm.basis[kAffRun + b];

    uint32_t rn = tile_base(first);
    chain_wait();  // everything above reads only the program
    for (uint32_t t = first; t < end; t += step) {
        const uint32_t r0 = rn;
        E x[kNR], y[kNR];
        {
            // the registers in Gray-code order: one XOR per address
            const uint32_t g[4] = {sm.basis[4], sm.basis[5], sm.basis[6], sm.basis[7]};
            uint32_t r = r0 ^ ra;
#pragma unroll
            for (int i = 0; i < kNR; i++) {
                const int j = i ^ (i >> 1);
                if (i) r ^= g[ctz_const(i)];
                x[j] = __ldcg(src + r);
                if constexpr (ADJ) y[j] = __ldcg(lam + r);
            }
        }
        if (t + step < end) {
            rn = tile_base(t + step);
            const uint32_t r = (rn ^ rp) & ~uint32_t(kRun - 1);
#pragma unroll
            for (int i = 0; i < int(sizeof(E)) / 8; i++) {
                prefetch_l2(src + r + i * (kRun / 2));
                if constexpr (ADJ) prefetch_l2(lam + r + i * (kRun / 2));
            }
        }
        // selector bits of the tile: lane s takes selectors s and s + 32
        const bool b0 = lane < nsel && (__popc(sm.alpha[lane] & r0) & 1);
        const bool b1 = lane + 32u < nsel && (__popc(sm.alpha[lane + 32u] & r0) & 1);
        const uint64_t P = uint64_t(__ballot_sync(0xffffffffu, b0)) | (uint64_t(__ballot_sync(0xffffffffu, b1)) << 32);
        const uint64_t c = P ^ lw;
        if (win0 || win1) {
            __syncthreads();  // the previous tile's polynomials and sums are read
            if (win0) window_eval(sm, ent0, w0, 0, P ^ lwe, tid & 15u, tid >> 4);
            if constexpr (!ADJ) {
                if (win1) window_eval(sm, ent1, w1, 1, P ^ lwe, tid & 15u, tid >> 4);
            }
            __syncthreads();
        }
        if (win0) {
            if constexpr (ADJ) window_grad(x, y, sm, w0, P, tid);
            window_apply<0, ADJ>(x, y, sm, w0.pairs, 0, lane, warp);
        }
        gates<4, ADJ, FORM>(x, y, mask, mu, refl, c, sm, tid);
        if (need_c) {
            exchange<0, 2, ADJ ? 2 : 1>(x, y, sm.slab, lane, warp);
            gates<0, ADJ, FORM>(x, y, mask, mu, refl, P ^ lw0, sm, tid);
            exchange<2, 1, ADJ ? 2 : 1>(x, y, sm.slab, lane, warp);
        } else if (need_b) {
            exchange<0, 1, ADJ ? 2 : 1>(x, y, sm.slab, lane, warp);
        }
        if (need_b) gates<8, ADJ, FORM>(x, y, mask, mu, refl, c, sm, tid);
        if constexpr (!ADJ) {
            if (win1) window_apply<1, false>(x, y, sm, w1.pairs, 1, lane, warp);
        }
        if (FORM == 2 && mask) {
            const RT f = (par64(c & neg_high) ^ par64((P ^ lw0) & neg_low)) ? -scale : scale;
#pragma unroll
            for (int j = 0; j < kNR; j++) {
                x[j] = scaled(f, x[j]);
                if constexpr (ADJ) y[j] = scaled(f, y[j]);
            }
        }
        {
            const uint32_t *gb = sm.basis + (need_b ? 8 : 4);
            const uint32_t g[4] = {gb[0], gb[1], gb[2], gb[3]};
            uint32_t r = r0 ^ (need_b ? rb : ra);
#pragma unroll
            for (int i = 0; i < kNR; i++) {
                const int j = i ^ (i >> 1);
                if (i) r ^= g[ctz_const(i)];
                __stcg(psi + r, x[j]);
                if constexpr (ADJ) __stcg(lam + r, y[j]);
            }
        }
    }
    if constexpr (ADJ) {
        __syncthreads();
        for (uint32_t i = tid; i < w0.nterms; i += kThreads)
            if (sm.term[i].gk) atomicAdd(&grads[sm.term[i].slot], sm.tacc[i]);
        // warp w sums gates w and w + 8
        for (uint32_t k = warp; k < uint32_t(kAffBits); k += kThreads / 32) {
            if (!((mask >> k) & 1u) || !sm.gen[k]) continue;
            double s = 0.0;
            for (int i = 0; i < kThreads / 32; i++) s += sm.gacc[k][i * 32 + int(lane)];
            s = warp_sum_f64(s);
            if (lane == 0) atomicAdd(&grads[p.gate[k].slot], s);
        }
    }
}

}  // namespace adev
}  // namespace zxh
