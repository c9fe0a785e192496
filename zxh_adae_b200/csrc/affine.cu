// affine.cu -- the affine tile pass (sm_100a): up to 12 commuting single-qubit gates with any
// pair deltas (the state after CX transport through the affine map), diagonal windows
// before and after them, in one read and one write of the state; in adjoint form on two
// states with every gradient reduced in FP64.
//
// The general strided pass (grow.cu) keeps one item's rows in a warp's registers, so it
// takes 4 gates whose deltas leave the low bits, and each lane evaluates every window term
// for its own few amplitudes: on the 24-qubit ansatz (RY, RZ, CX chain) 5 passes a layer,
// bound by instruction issue (2700 us forward, 130 us per reverse pass where the two states
// move in 80 us). Here a CTA works on a tile of 2^12 amplitudes r0 ^ span(basis): four basis
// vectors span the low 4 real bits (runs of 16 contiguous amplitudes: 128 bytes complex64,
// 256 complex128), the other eight are pair deltas, so 8 gates ride whatever bits their
// deltas span, plus the up to 4 inside the run, and a 24-gate layer takes 3 passes. The
// amplitudes move between register layouts through shared memory:
//     A  registers 4..7    lanes 0..3, 8  warps 9..11   (loads)
//     B  registers 8..11   lanes 0..4     warps 5..7    (stores)
//     C  registers 0..3    lanes 4..8     warps 9..11
// A pass runs A, A -> B or A -> C -> B as its gates need. A selector of the map flips with
// one of the eight deltas at most (they are pair deltas of distinct qubits), so a window
// is a polynomial of degree two in eight bits whose coefficients depend only on the tile
// and the position in the run: the CTA evaluates the terms 16 times per tile (once per run
// position) instead of once per thread, and a thread reads the polynomial from shared
// memory. Real addresses are 32-bit (states of at most 2^32 amplitudes; larger ones take the
// general strided passes). Gradients of window terms come from the marginals of w = Im(conj(lambda) psi) over
// the same bits, reduced once per tile. Exchanges to and from C put tile index i in slot
// i ^ (bits 4..7 of i), the others in slot i: either way the lanes that share a bank cycle
// cover one 128-byte row.
//
// Measured on that ansatz, complex64: 24 forward passes, 1.33 ms (46 and 2.60 ms as general
// strided passes), 50 us a pass without a window; reverse 126 us a pass, the gradient 5.3
// instead of 9.9 ms. Three CTAs an SM forward (80 registers; four at 64: 54 us a pass), two
// in the adjoint form, which fills the registers with two states; issue is then at 31 to
// 50 %, DRAM at 33 to 45 % with half the state in L2: latency between barriers is left.
#include "affine_dev.cuh"

#include <algorithm>
#include <cuda_runtime.h>

namespace zxh {

namespace {

using namespace adev;

template <typename E, bool ADJ, int FORM>
__global__ void __launch_bounds__(kThreads, sizeof(E) == 8 ? (ADJ ? 2 : 3) : (ADJ ? 1 : 2))
    affine_kernel(const uint8_t *__restrict__ blob, uint64_t poff, uint64_t toff, E *psi, const E *src, E *lam,
                  double *grads, uint64_t ntiles)
{
    extern __shared__ __align__(128) unsigned char s_raw[];
    chain_trigger();
    affine_body<E, ADJ, FORM>(*reinterpret_cast<AffSmem<E, ADJ> *>(s_raw), blob, poff, toff, psi, src, lam, grads,
                              blockIdx.x, gridDim.x, uint32_t(ntiles));
}

template <typename E, bool ADJ, int FORM>
cudaError_t launch_affine(const uint8_t *blob, uint64_t poff, uint64_t toff, uint64_t ntiles, E *psi, const E *src, E *lam,
                          double *grads, bool chained, int sms, cudaStream_t st)
{
    auto kern = affine_kernel<E, ADJ, FORM>;
    const int smem = int(sizeof(AffSmem<E, ADJ>));
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, size_t(smem));
    const unsigned grid = unsigned(std::min<uint64_t>(ntiles, uint64_t(sms) * uint64_t(std::max(1, per_sm))));
    return launch_chained(chained, kern, grid, kThreads, size_t(smem), st, blob, poff, toff, psi,
                          src ? src : static_cast<const E *>(psi), lam, grads, ntiles);
}

template <typename E, bool ADJ, typename... A>
cudaError_t affine_form(int form, A... args)
{
    switch (form) {
    case 0: return launch_affine<E, ADJ, 0>(args...);
    case 1: return launch_affine<E, ADJ, 1>(args...);
    default: return launch_affine<E, ADJ, 2>(args...);
    }
}

template <typename E>
cudaError_t affine_typed(int form, const uint8_t *blob, uint64_t poff, uint64_t toff, uint64_t ntiles, E *psi, const E *src,
                         E *lam, double *grads, bool chained, int sms, cudaStream_t st)
{
    return lam ? affine_form<E, true>(form, blob, poff, toff, ntiles, psi, src, lam, grads, chained, sms, st)
               : affine_form<E, false>(form, blob, poff, toff, ntiles, psi, src, lam, grads, chained, sms, st);
}

}  // namespace

cudaError_t run_affine(const uint8_t *dblob, uint64_t poff, uint64_t toff, uint64_t ntiles, int elem_bytes, int form,
                       void *psi, const void *psi_src, void *lam, double *grads, bool chained, int sms, cudaStream_t st)
{
    if (elem_bytes == 8)
        return affine_typed(form, dblob, poff, toff, ntiles, static_cast<float2 *>(psi),
                            static_cast<const float2 *>(psi_src), static_cast<float2 *>(lam), grads, chained, sms, st);
    return affine_typed(form, dblob, poff, toff, ntiles, static_cast<double2 *>(psi),
                        static_cast<const double2 *>(psi_src), static_cast<double2 *>(lam), grads, chained, sms, st);
}

}  // namespace zxh
