// permute.cu -- get_state on the device (sm_100a): the state in real-address order
// becomes the 2^N amplitudes in virtual order (optionally bit-reversed, zxh.cpp:
// 579-636 of ZXH-Sim), times the global phase.
//
// out[B r ^ b] = phase * state[r] with B linear over GF(2) (the affine map with its
// rows reversed for the reference's order), so neighbouring real addresses land far
// apart: written one amplitude at a time every 8- or 16-byte store touches its own
// 32-byte sector of DRAM, and a bit reversal of 2^27 complex64 amplitudes took 6.6 ms
// (0.33 TB/s). The pass is bound by memory only if both sides run over contiguous
// pieces, so a CTA takes a tile closed under both: the cosets of
//     V = span(e_0 .. e_{c-1}, g_0 .. g_{k-1}),
// e_i the low real bits and g_i the real vectors whose images lie in the low c bits of
// the output index (k = c when the map is square). It reads V as runs of 2^c
// contiguous amplitudes, turns it in shared memory and writes runs of 2^c contiguous
// amplitudes. c = 6 (complex64) and 5 (complex128), runs of 512 bytes, and tiles of 2^12 and
// 2^11 amplitudes, 32 KiB: registers leave room for two and three CTAs an SM (124 and 80 a
// thread), and one CTA's reads overlap another's writes. Every index is an XOR of per-bit
// vectors computed on the host.
// 2^27 complex64 amplitudes: 0.387 ms, 5.55 TB/s (0.86 of the measured copy).
#include "core.h"
#include "dev.cuh"
#include "permute.h"

#include <algorithm>
#include <cuda_runtime.h>

namespace zxh {

namespace {

template <typename E>
struct PermCfg;
template <>
struct PermCfg<float2> {
    static constexpr int C = 6, D = 12, BANK = 4;  // run bits, tile bits, index bits of a 128-byte row
};
template <>
struct PermCfg<double2> {
    static constexpr int C = 5, D = 11, BANK = 3;
};

template <typename E>
__device__ __forceinline__ E perm_phase(E a, decltype(E{}.x) gr, decltype(E{}.x) gi)
{
    E o;
    o.x = a.x * gr - a.y * gi;
    o.y = a.x * gi + a.y * gr;
    return o;
}

// NS: tile entries per thread.
template <typename E, int NS>
__global__ void __launch_bounds__(kThreads) permute_kernel(const E *__restrict__ state, E *__restrict__ out,
                                                           const __grid_constant__ PermDev p, double gre, double gim)
{
    using R = decltype(E{}.x);
    __shared__ E slab[NS * kThreads];
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const bool on = tid < (1u << p.d);
    uint64_t rt = 0, wt = 0;
    uint32_t st = 0, mt = 0;
#pragma unroll
    for (int b = 0; b < 8; b++)
        if ((tid >> b) & 1u) {
            rt ^= p.rvec[b];
            st ^= p.spos[b];
            wt ^= p.wimg[b];
            mt ^= p.wpos[b];
        }
    const uint64_t tr0 = p.tr[lane], tr1 = p.tr[lane + 32u], ti0 = p.ti[lane], ti1 = p.ti[lane + 32u];
    const R gr = R(gre), gi = R(gim);
    for (uint64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
        // lane j holds tile bits j and j + 32
        const bool b0 = (t >> lane) & 1u, b1 = (t >> (lane + 32u)) & 1u;
        const uint64_t rl = (b0 ? tr0 : 0) ^ (b1 ? tr1 : 0);
        const uint64_t il = (b0 ? ti0 : 0) ^ (b1 ? ti1 : 0);
        const uint64_t r0 = (uint64_t(__reduce_xor_sync(0xffffffffu, uint32_t(rl >> 32))) << 32) |
                            __reduce_xor_sync(0xffffffffu, uint32_t(rl));
        const uint64_t i0 = (uint64_t(__reduce_xor_sync(0xffffffffu, uint32_t(il >> 32))) << 32) |
                            __reduce_xor_sync(0xffffffffu, uint32_t(il));
        E x[NS];
#pragma unroll
        for (int s = 0; s < NS; s++) {
            uint64_t r = r0 ^ rt;
#pragma unroll
            for (int b = 0; (1 << b) < NS; b++)
                if ((s >> b) & 1) r ^= p.rvec[8 + b];
            if (on) x[s] = __ldcs(state + r);
        }
        __syncthreads();  // the previous tile has been read out of the slab
#pragma unroll
        for (int s = 0; s < NS; s++) {
            uint32_t q = st;
#pragma unroll
            for (int b = 0; (1 << b) < NS; b++)
                if ((s >> b) & 1) q ^= p.spos[8 + b];
            if (on) slab[q] = x[s];
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < NS; s++) {
            uint32_t q = mt;
            uint64_t w = i0 ^ wt;
#pragma unroll
            for (int b = 0; (1 << b) < NS; b++)
                if ((s >> b) & 1) {
                    q ^= p.wpos[8 + b];
                    w ^= p.wimg[8 + b];
                }
            if (on) __stcs(out + (w ^ p.b), perm_phase(slab[q], gr, gi));
        }
    }
}

// Maps whose columns are dependent (a CX whose control is its target): several real
// addresses share an output, one amplitude at a time.
template <typename E>
__global__ void __launch_bounds__(kThreads) scatter_kernel(const E *__restrict__ state, uint64_t n_real,
                                                           const __grid_constant__ PermCols c, double gre, double gim,
                                                           E *__restrict__ out)
{
    using R = decltype(E{}.x);
    const R gr = R(gre), gi = R(gim);
    for (uint64_t r = uint64_t(blockIdx.x) * kThreads + threadIdx.x; r < n_real; r += uint64_t(gridDim.x) * kThreads) {
        uint64_t v = c.b;
        for (int j = 0; j < c.m; j++)
            if ((r >> j) & 1) v ^= c.col[j];
        out[v] = perm_phase(state[r], gr, gi);
    }
}

template <typename E, int NS>
cudaError_t launch_permute(const E *state, E *out, const PermDev &p, double gre, double gim, int sms, cudaStream_t st)
{
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, permute_kernel<E, NS>, kThreads, 0);
    const unsigned grid = unsigned(std::min<uint64_t>(p.ntiles, uint64_t(sms) * uint64_t(std::max(1, per_sm))));
    permute_kernel<E, NS><<<grid, kThreads, 0, st>>>(state, out, p, gre, gim);
    return cudaGetLastError();
}

template <typename E>
cudaError_t permute_typed(const void *state, const PermCols &c, double gre, double gim, void *out, int sms,
                          cudaStream_t st)
{
    auto *src = static_cast<const E *>(state);
    auto *dst = static_cast<E *>(out);
    PermDev p;
    if (!perm_plan(c, PermCfg<E>::C, PermCfg<E>::D, PermCfg<E>::BANK, p)) {
        const uint64_t n_real = 1ULL << c.m;
        const unsigned grid = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((n_real + kThreads - 1) / kThreads,
                                                                                uint64_t(sms) * 16)));
        scatter_kernel<E><<<grid, kThreads, 0, st>>>(src, n_real, c, gre, gim, dst);
        return cudaGetLastError();
    }
    switch (p.d <= 8 ? 0 : int(p.d) - 8) {
    case 0: return launch_permute<E, 1>(src, dst, p, gre, gim, sms, st);
    case 1: return launch_permute<E, 2>(src, dst, p, gre, gim, sms, st);
    case 2: return launch_permute<E, 4>(src, dst, p, gre, gim, sms, st);
    case 3: return launch_permute<E, 8>(src, dst, p, gre, gim, sms, st);
    default: return launch_permute<E, 16 / (sizeof(E) / 8)>(src, dst, p, gre, gim, sms, st);
    }
}

}  // namespace

cudaError_t run_permute(const void *state, const PermCols &cols, double gre, double gim, void *out, int elem_bytes,
                        int sms, cudaStream_t st)
{
    return elem_bytes == 8 ? permute_typed<float2>(state, cols, gre, gim, out, sms, st)
                           : permute_typed<double2>(state, cols, gre, gim, out, sms, st);
}

}  // namespace zxh
