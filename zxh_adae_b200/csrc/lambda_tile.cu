// lambda_tile.cu -- lambda = H psi and <psi|H|psi> over tiles held in shared memory
// (sm_100a), for states of at least 2^12 amplitudes and all but a few terms.
//
// H is a sum of Z, ZZ and X terms (lambda_dev.cuh has the real-address forms). An X term
// reads psi[r ^ delta]; done as one gather per term over the whole state that is one more
// read of the state each: 24 terms on 2^24 complex64 amplitudes took 0.49 ms where one
// read of the state takes 0.02 (bound by L2), and 9.7 ms at 2^28 (bound by DRAM). Here a
// CTA holds a tile closed under the flips it applies: 2^12 amplitudes r0 ^ span(basis),
// the basis vectors being a basis of the low 4 real bits (runs of 16 contiguous
// amplitudes) and up to 8 flips that are independent modulo them (any real bits, as after
// CX transport). One read of the state then serves up to 12 X terms, so a chain of 24
// takes 3 passes; the Z and ZZ terms ride in the first.
//
// Tile coordinates 0..3: lanes 0..3; 4..7: a thread's 16 registers; 8: lane bit 4; 9..11:
// the warp. A flip of a register coordinate is another register; of the others, a read of
// the tile in shared memory, whose 16 lanes cover one 128-byte row either way, so every
// access is conflict-free. A pass is bound by the shared-memory reads (8 per amplitude of a
// full low pass) and instruction issue: 24 terms take 0.17 ms at 2^24 and 2.9 ms at 2^28
// complex64 amplitudes, 0.30 and 5.2 ms in complex128 (one CTA an SM).
//
// The diagonal sum at a thread's 16 amplitudes is the Walsh-Hadamard transform over the
// register bits of the coefficients summed by register part (the host sorts the terms by
// it); a term's sign outside the registers is one bit per tile (one parity per term) XOR
// one per thread.
#include "adjoint.h"
#include "chain.cuh"
#include "core.h"
#include "dev.cuh"

#include <algorithm>
#include <cuda_runtime.h>
#include <vector>

namespace zxh {

namespace {

constexpr int kLamT = 12, kLamRun = 4, kLamRegs = 16;

template <typename E>
struct LamSmem {
    using R = typename ET<E>::R;
    E slab[1 << kLamT];
    uint64_t mask[kMaxTerms];
    R coef[kMaxTerms];
    uint32_t thread_sign[kMaxTerms / 32][kThreads];
    uint32_t tile_sign[2][kMaxTerms / 32];
    double red[kThreads / 32];
};

// c x + y, one paired FP32 FMA or two FP64 ones
__device__ __forceinline__ float2 axpy(float c, float2 x, float2 y) { return __ffma2_rn(make_float2(c, c), x, y); }
__device__ __forceinline__ double2 axpy(double c, double2 x, double2 y)
{
    return make_double2(fma(c, x.x, y.x), fma(c, x.y, y.y));
}

// c, negated where bit 0 of s is set
__device__ __forceinline__ float flip_sign(float c, uint32_t s) { return __uint_as_float(__float_as_uint(c) ^ (s << 31)); }
__device__ __forceinline__ double flip_sign(double c, uint32_t s)
{
    return __hiloint2double(__double2hiint(c) ^ int(s << 31), __double2loint(c));
}

// MODE 0: energy only; 1: lam is written; 2: lam is added to. With lam the energy comes from
// the whole of it, in the last pass (last != 0).
template <typename E, int MODE>
__global__ void __launch_bounds__(kThreads, sizeof(E) == 8 ? (MODE == 0 ? 3 : 2) : 1)
    lambda_tile_kernel(const E *psi, E *lam, const __grid_constant__ LamPassDev p,
                       const TermDev *__restrict__ terms, double *energy, int last)
{
    using R = typename ET<E>::R;
    extern __shared__ __align__(128) unsigned char s_raw[];
    LamSmem<E> &sm = *reinterpret_cast<LamSmem<E> *>(s_raw);
    chain_trigger();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t nd = p.nd;

    // this thread's part of the address and of the tile index
    uint64_t rt = 0;
#pragma unroll
    for (int b = 0; b < 5; b++)
        if ((lane >> b) & 1u) rt ^= p.basis[b < 4 ? b : 8];
#pragma unroll
    for (int b = 0; b < 3; b++)
        if ((warp >> b) & 1u) rt ^= p.basis[9 + b];
    const uint32_t it = (lane & 15u) | ((lane >> 4) << 8) | (warp << 9);
    const uint64_t tr0 = p.tr[lane], tr1 = p.tr[lane + 32u];

    if (tid < nd) {
        const TermDev t = terms[p.diag0 + tid];
        const bool zz = t.kind == 2;
        sm.mask[tid] = zz ? t.a0 ^ t.a1 : t.a0;
        sm.coef[tid] = ((zz ? t.b0 ^ t.b1 : t.b0) & 1u) ? -R(t.coef) : R(t.coef);
    }
    __syncthreads();
    for (uint32_t w = 0; w * 32u < nd; w++) {
        uint32_t bits = 0;
        for (uint32_t k = 0; k < 32u && w * 32u + k < nd; k++) bits |= uint32_t(par64(sm.mask[w * 32u + k] & rt)) << k;
        sm.thread_sign[w][tid] = bits;
    }

    auto tile_base = [&](uint64_t t) {
        const uint64_t rl = (((t >> lane) & 1u) ? tr0 : 0) ^ (((t >> (lane + 32u)) & 1u) ? tr1 : 0);
        return (uint64_t(__reduce_xor_sync(0xffffffffu, uint32_t(rl >> 32))) << 32) |
               __reduce_xor_sync(0xffffffffu, uint32_t(rl));
    };
    // the run of 16 amplitudes this thread asks L2 for, one tile ahead
    uint64_t rp = 0;
#pragma unroll
    for (int b = 0; b < kLamT - kLamRun; b++)
        if ((tid >> b) & 1u) rp ^= p.basis[kLamRun + b];

    double en = 0.0;
    uint32_t turn = 0;
    uint64_t rn = tile_base(blockIdx.x);
    chain_wait();  // everything above reads only the terms
    for (uint64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x, turn ^= 1u) {
        const uint64_t r0 = rn;
        const uint64_t ra = r0 ^ rt;
        auto addr = [&](int j) {
            uint64_t r = ra;
#pragma unroll
            for (int b = 0; b < 4; b++)
                if ((j >> b) & 1) r ^= p.basis[4 + b];
            return r;
        };
        E x[kLamRegs], l[kLamRegs];
#pragma unroll
        for (int j = 0; j < kLamRegs; j++) {
            x[j] = __ldcg(psi + addr(j));
            if constexpr (MODE == 2) l[j] = __ldcg(lam + addr(j));
        }
        if (t + gridDim.x < p.ntiles) {
            rn = tile_base(t + gridDim.x);
            const uint64_t r = (rn ^ rp) & ~uint64_t((1 << kLamRun) - 1);
#pragma unroll
            for (int i = 0; i < int(sizeof(E)) / 8; i++) {
                prefetch_l2(psi + r + i * (1 << kLamRun) / 2);
                if constexpr (MODE == 2) prefetch_l2(lam + r + i * (1 << kLamRun) / 2);
            }
        }
        if (warp * 32u < nd) {
            const uint32_t k = tid;
            const uint32_t bits = __ballot_sync(0xffffffffu, k < nd && par64(sm.mask[k] & r0));
            if (lane == 0) sm.tile_sign[turn][warp] = bits;
        }
        __syncthreads();  // the slab's previous reads are done
#pragma unroll
        for (int j = 0; j < kLamRegs; j++) sm.slab[it | uint32_t(j << 4)] = x[j];
        __syncthreads();

        // diagonal part (the first pass): coefficients by register part, then the transform
        if (MODE != 2 && nd) {
            R u[kLamRegs];
            uint32_t word = ~0u, signs = 0;
#pragma unroll
            for (int g = 0; g < kLamRegs; g++) {
                R a = 0;
                for (uint32_t k = p.goff[g]; k < p.goff[g + 1]; k++) {
                    if (k >> 5 != word) {
                        word = k >> 5;
                        signs = sm.tile_sign[turn][word] ^ sm.thread_sign[word][tid];
                    }
                    a += flip_sign(sm.coef[k], signs >> (k & 31u));
                }
                u[g] = a;
            }
#pragma unroll
            for (int b = 1; b < kLamRegs; b <<= 1)
#pragma unroll
                for (int g = 0; g < kLamRegs; g++)
                    if (!(g & b)) {
                        const R lo = u[g], hi = u[g | b];
                        u[g] = lo + hi;
                        u[g | b] = lo - hi;
                    }
#pragma unroll
            for (int j = 0; j < kLamRegs; j++) {
                l[j].x = u[j] * x[j].x;
                l[j].y = u[j] * x[j].y;
            }
        } else if (MODE != 2) {
#pragma unroll
            for (int j = 0; j < kLamRegs; j++) l[j].x = l[j].y = R(0);
        }
        // flips of register coordinates
#pragma unroll
        for (int b = 0; b < 4; b++) {
            if (!((p.xmask >> (4 + b)) & 1u)) continue;
            const R c = R(p.xc[4 + b]);
#pragma unroll
            for (int j = 0; j < kLamRegs; j++) l[j] = axpy(c, x[j ^ (1 << b)], l[j]);
        }
        // flips of lane and warp coordinates
#pragma unroll
        for (int k = 0; k < kLamT; k++) {
            if ((k >= 4 && k < 8) || !((p.xmask >> k) & 1u)) continue;
            const R c = R(p.xc[k]);
            const E *row = sm.slab + (it ^ (1u << k));
#pragma unroll
            for (int j = 0; j < kLamRegs; j++) l[j] = axpy(c, row[j << 4], l[j]);
        }
        if (MODE == 0 || last) {
#pragma unroll
            for (int j = 0; j < kLamRegs; j++)  // Re(conj(psi) lambda)
                en += double(x[j].x) * double(l[j].x) + double(x[j].y) * double(l[j].y);
        }
        if constexpr (MODE != 0) {
#pragma unroll
            for (int j = 0; j < kLamRegs; j++) __stcg(lam + addr(j), l[j]);
        }
    }
    if (MODE != 0 && !last) return;
    en = warp_sum_f64(en);
    if (lane == 0) sm.red[warp] = en;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < kThreads / 32; w++) s += sm.red[w];
        atomicAdd(energy, s);
    }
}

template <typename E, int MODE>
cudaError_t launch_pass(const E *psi, E *lam, const LamPassDev &p, const TermDev *terms, double *energy, bool last,
                        bool chained, int sms, cudaStream_t st)
{
    auto kern = lambda_tile_kernel<E, MODE>;
    const int smem = int(sizeof(LamSmem<E>));
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, size_t(smem));
    const unsigned grid = unsigned(std::min<uint64_t>(p.ntiles, uint64_t(sms) * uint64_t(std::max(1, per_sm))));
    return launch_chained(chained, kern, grid, kThreads, size_t(smem), st, psi, lam, p, terms, energy, last ? 1 : 0);
}

template <typename E>
cudaError_t lambda_tiles_typed(const E *psi, E *lam, const std::vector<LamPassDev> &passes, const TermDev *terms,
                               double *energy, int sms, cudaStream_t st)
{
    for (size_t i = 0; i < passes.size(); i++) {
        const bool last = i + 1 == passes.size();
        const cudaError_t e = !lam ? launch_pass<E, 0>(psi, lam, passes[i], terms, energy, last, i > 0, sms, st)
                              : i  ? launch_pass<E, 2>(psi, lam, passes[i], terms, energy, last, i > 0, sms, st)
                                   : launch_pass<E, 1>(psi, lam, passes[i], terms, energy, last, i > 0, sms, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int top_bit(uint64_t x) { return 63 - __builtin_clzll(x); }

}  // namespace

// Where lambda_kernel's one gather per X term and one parity per amplitude and Z term beat the
// tiles, whose tables, slab and barriers cost the same for one term as for many. A few Z terms
// of 28 qubits: complex128 1 term 0.59 against 1.09 ms, 4 terms 0.65 / 1.43, 12 terms 1.47 / 1.66,
// 16 terms 1.87 / 1.69; complex64 1 term 0.51 / 0.65, 4 terms 0.68 / 0.71, 6 terms 0.83 / 0.73.
// One X term more is a read of the state (28 qubits complex64 0.82 / 0.44), but nothing while
// the setup bounds both: at 16 qubits complex64 1 X and 8 Z terms take 10 against 13 us, 3 X and
// 12 Z 12 and 13; at 22 qubits complex128 1 X and 4 Z 27 against 32.
static bool gather_terms(size_t nx, size_t nd, int m, int elem_bytes)
{
    if (m <= 18) return nx <= 1 ? nd <= 32 : nx == 2 && nd <= 12;
    if (nx == 0) return nd <= (elem_bytes == 8 ? 4 : 12);
    return elem_bytes == 16 && m <= 22 && nx == 1 && nd >= 1 && nd <= 4;
}

std::vector<LamPassDev> plan_lambda(std::vector<TermDev> &terms, int m, int elem_bytes)
{
    std::vector<LamPassDev> out;
    size_t nx = 0;
    while (nx < terms.size() && terms[nx].kind == 3) nx++;
    if (m < kLamT || gather_terms(nx, terms.size() - nx, m, elem_bytes)) return out;
    struct Flip { uint64_t delta; double coef; };
    std::vector<Flip> flips;
    for (nx = 0; nx < terms.size() && terms[nx].kind == 3;) {
        const TermDev &t = terms[nx++];
        auto same = std::find_if(flips.begin(), flips.end(), [&](const Flip &f) { return f.delta == t.delta; });
        if (same != flips.end()) same->coef += t.coef;
        else flips.push_back({t.delta, t.coef});
    }
    // flips of low bits first: the first tiles are then whole runs of memory
    std::stable_sort(flips.begin(), flips.end(), [](const Flip &a, const Flip &b) { return a.delta < b.delta; });

    auto reduced = [](uint64_t v, const std::vector<uint64_t> &ech) {
        for (uint64_t b : ech)
            if ((v >> top_bit(b)) & 1) v ^= b;
        return v;
    };
    auto insert = [](uint64_t v, std::vector<uint64_t> &ech) {
        ech.push_back(v);
        std::sort(ech.rbegin(), ech.rend());
    };
    do {
        LamPassDev p = {};
        std::vector<uint64_t> low, high;  // echelon forms of the low parts and of the high parts
        int nlow = 0, nhigh = 0;
        std::vector<Flip> rest;
        for (const Flip &f : flips) {
            const bool inside = (f.delta >> kLamRun) == 0;
            std::vector<uint64_t> &ech = inside ? low : high;
            const uint64_t v = reduced(inside ? f.delta : f.delta >> kLamRun, ech);
            const bool room = inside ? nlow < kLamRun : nhigh < kLamT - kLamRun;
            if (!v || !room) {
                rest.push_back(f);
                continue;
            }
            insert(v, ech);
            const int k = inside ? nlow++ : kLamRun + nhigh++;
            p.basis[k] = f.delta;
            p.xc[k] = f.coef;
            p.xmask |= 1u << k;
        }
        flips.swap(rest);
        for (int b = 0; b < m; b++) {  // complete the basis by single bits, the lowest first
            const bool inside = b < kLamRun;
            std::vector<uint64_t> &ech = inside ? low : high;
            if (inside ? nlow == kLamRun : nhigh == kLamT - kLamRun) continue;
            const uint64_t v = reduced(inside ? 1ULL << b : 1ULL << (b - kLamRun), ech);
            if (!v) continue;
            insert(v, ech);
            p.basis[inside ? nlow++ : kLamRun + nhigh++] = 1ULL << b;
        }
        uint64_t piv = low_mask(kLamRun);
        for (uint64_t v : high) piv |= 1ULL << (top_bit(v) + kLamRun);
        int t = 0;
        for (int b = 0; b < m; b++)
            if (!((piv >> b) & 1)) p.tr[t++] = 1ULL << b;
        p.ntiles = 1ULL << t;
        if (out.empty()) {
            p.diag0 = uint32_t(nx);
            p.nd = uint32_t(terms.size() - nx);
            auto part = [&](const TermDev &d) {
                const uint64_t mask = d.kind == 2 ? d.a0 ^ d.a1 : d.a0;
                uint32_t g = 0;
                for (int b = 0; b < 4; b++) g |= uint32_t(parity64(mask & p.basis[4 + b])) << b;
                return g;
            };
            std::stable_sort(terms.begin() + long(nx), terms.end(),
                             [&](const TermDev &a, const TermDev &b) { return part(a) < part(b); });
            for (size_t i = nx; i < terms.size(); i++) p.goff[part(terms[i]) + 1]++;
            for (int g = 0; g < kLamRegs; g++) p.goff[g + 1] += p.goff[g];
        }
        out.push_back(p);
    } while (!flips.empty());
    return out;
}

cudaError_t run_lambda_tiles(const void *psi, void *lam, int elem_bytes, const std::vector<LamPassDev> &passes,
                             const TermDev *dterms, double *energy, int sms, cudaStream_t st)
{
    if (elem_bytes == 8)
        return lambda_tiles_typed(static_cast<const float2 *>(psi), static_cast<float2 *>(lam), passes, dterms, energy,
                                  sms, st);
    return lambda_tiles_typed(static_cast<const double2 *>(psi), static_cast<double2 *>(lam), passes, dterms, energy, sms,
                              st);
}

}  // namespace zxh
