// sampler.cu -- multinomial sampler of the B200-native ZXH path (sm_100a).
//
// Draws the same outcomes as the reference GPU sampler when fed the same seed: it
// consumes the reference's uniform stream (splitmix64 of seed-mixed shot and output
// indices, src/zxh/src/measure/measure_cuda.cu:387-443,493-515) with the same two-
// level structure (segments of 2^12 amplitudes, then an offset inside the segment),
// and returns shots grouped by segment in the reference's output order. The
// machinery is new:
//   seg_mass_kernel      one streaming read of the state: per-segment FP64 |amp|^2
//                        mass, one warp per segment (and the 32 lane-range masses of
//                        each segment, kept for the resolve step).
//   mass scan (3 kernels) inclusive FP64 scan of the masses: the segment CDF (the
//                        reference runs segment_mass_kernel + a CUB scan).
//   count_kernel         shot -> segment by binary search, warp-aggregated atomics.
//   offsets (3 kernels)  exclusive scan of the per-segment counts.
//   small_draw_kernel    the three steps above in one CTA, for few segments and shots.
//   resolve_warp_kernel  segments hit by <= 32 shots: one warp streams the segment
//                        once, lane-scans it and places each shot with a warp-
//                        cooperative search (ballot over lane prefixes, then over
//                        4-amplitude sub-ranges).
//   resolve_cta_kernel   heavier segments, one per CTA (round robin): the CTA builds
//                        the segment CDF in shared memory and binary-searches it.
//   map_kernel           real index -> packed virtual bits (measure_cuda.cu:315-338).
// No kernel waits on another CTA.
#include "chain.cuh"
#include "core.h"
#include "dev.cuh"
#include "permute.h"
#include "sampler.h"

#include <algorithm>
#include <cuda_runtime.h>

namespace zxh {

namespace {

constexpr uint64_t kSeedShot = 0x510e527fade682d1ULL;    // measure_cuda.cu:427
constexpr uint64_t kSeedOffset = 0x9b05688c2b3e6c1fULL;  // measure_cuda.cu:499
constexpr int kWarpMax = 32;
constexpr int kScanBlock = 4096;

__device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
    uint64_t z = x + 0x9e3779b97f4a7c15ULL;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

// (mant + 1) / (2^53 + 1) evaluated in double; 2^53 + 1 rounds to 2^53 as on the
// reference device (measure_cuda.cu:395-410).
__device__ __forceinline__ double uniform_open01(uint64_t seed)
{
    const uint64_t mant = splitmix64(seed) >> 11;
    return (static_cast<double>(mant) + 1.0) / (static_cast<double>(1ULL << 53) + 1.0);
}

template <typename E>
__device__ __forceinline__ double prob(const E &a)
{
    const double re = double(a.x), im = double(a.y);
    return re * re + im * im;
}


// |amp|^2 mass of seg[lo, hi), in order; complex64 ranges with even bounds use
// 16-byte loads.
__device__ __forceinline__ double range_mass(const float2 *seg, uint32_t lo, uint32_t hi)
{
    double part = 0.0;
    if (!((lo | hi) & 1)) {
        const float4 *v = reinterpret_cast<const float4 *>(seg);
        for (uint32_t k = lo / 2; k < hi / 2; k++) {
            const float4 x = __ldg(v + k);
            part += double(x.x) * x.x + double(x.y) * x.y;
            part += double(x.z) * x.z + double(x.w) * x.w;
        }
        return part;
    }
    for (uint32_t k = lo; k < hi; k++) part += prob(seg[k]);
    return part;
}

__device__ __forceinline__ double range_mass(const double2 *seg, uint32_t lo, uint32_t hi)
{
    double part = 0.0;
    for (uint32_t k = lo; k < hi; k++) part += prob(__ldg(seg + k));
    return part;
}

// ---------------------------------------------------------------------------

// Mass of lane l's range [l p, (l + 1) p) of a full 4096-amplitude segment, p =
// 128, read coalesced: in step g the warp reads 32 consecutive 16-byte vectors,
// which all belong to range g / G (G steps per range), and the range's mass is
// the warp's sum of them; lane l keeps range l. The same code runs in the segment
// pass and in the resolve step's fallback, so both see the same numbers.
__device__ __forceinline__ double vec_mass(const float4 &x)
{
    return (double(x.x) * x.x + double(x.y) * x.y) + (double(x.z) * x.z + double(x.w) * x.w);
}
__device__ __forceinline__ double vec_mass(const double2 &x) { return x.x * x.x + x.y * x.y; }

template <typename E>
__device__ __forceinline__ double lane_range_mass(const E *seg, int lane)
{
    using VT = typename ET<E>::VT;
    constexpr int G = 4096 / ET<E>::V / 32 / 32;  // steps per range: 2 (complex64), 4 (complex128)
    const VT *v = reinterpret_cast<const VT *>(seg);
    double mine = 0.0;
#pragma unroll 4
    for (int r = 0; r < 32; r++) {
        VT x[G];
#pragma unroll
        for (int i = 0; i < G; i++) x[i] = __ldcs(v + (r * G + i) * 32 + lane);
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < G; i++) t += vec_mass(x[i]);
        t = warp_sum_f64(t);
        if (lane == r) mine = t;
    }
    return mine;
}

// Lane l of a warp owns amplitudes [l p, (l + 1) p) of a segment, p = seglen / 32
// rounded up; its mass and the warp's inclusive prefix over lanes. The segment
// kernel and the resolve kernel both use this order, so a segment's total and its
// lane prefixes are the same numbers in both.
__device__ __forceinline__ double lane_prefix(double part, int lane)
{
    double incl = part;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    return incl;
}

// Per-segment FP64 mass, one warp per segment: one streaming read of the state.
// With parts, every lane's range mass is kept for the resolve step.
template <typename E>
__global__ void __launch_bounds__(kThreads) seg_mass_kernel(const E *__restrict__ state, uint64_t nseg, uint32_t seglen,
                                                            double *__restrict__ mass, double *__restrict__ parts)
{
    const int lane = threadIdx.x & 31;
    const uint64_t w0 = (uint64_t(blockIdx.x) * kThreads + threadIdx.x) >> 5;
    const uint64_t nw = (uint64_t(gridDim.x) * kThreads) >> 5;
    const uint32_t per_lane = (seglen + 31) / 32;
    const uint32_t lo = min(seglen, uint32_t(lane) * per_lane), hi = min(seglen, lo + per_lane);
    for (uint64_t sg = w0; sg < nseg; sg += nw) {
        const double part = seglen == 4096 ? lane_range_mass(state + sg * seglen, lane)
                                           : range_mass(state + sg * seglen, lo, hi);
        if (parts) parts[sg * 32 + uint64_t(lane)] = part;
        const double total = __shfl_sync(0xffffffffu, lane_prefix(part, lane), 31);
        if (lane == 0) mass[sg] = total;
    }
}

// The same masses, one CTA per full segment, for states whose segments are fewer than the
// chip's warps: a warp alone reads its 32 to 64 KiB in 32 steps one after another (25 us
// at 20 qubits complex128), eight of them share the ranges. Every range is summed as
// above, so the numbers are the same.
template <typename E>
__global__ void __launch_bounds__(kThreads) seg_mass_cta_kernel(const E *__restrict__ state, uint64_t nseg,
                                                                double *__restrict__ mass, double *__restrict__ parts)
{
    using VT = typename ET<E>::VT;
    constexpr int G = 4096 / ET<E>::V / 32 / 32, PER = 32 / (kThreads / 32);
    __shared__ double s_part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    chain_trigger();
    for (uint64_t sg = blockIdx.x; sg < nseg; sg += gridDim.x) {
        const VT *v = reinterpret_cast<const VT *>(state + sg * 4096);
        VT x[PER][G];
#pragma unroll
        for (int r = 0; r < PER; r++)
#pragma unroll
            for (int i = 0; i < G; i++) x[r][i] = __ldcs(v + ((warp * PER + r) * G + i) * 32 + lane);
#pragma unroll
        for (int r = 0; r < PER; r++) {
            double t = 0.0;
#pragma unroll
            for (int i = 0; i < G; i++) t += vec_mass(x[r][i]);
            t = warp_sum_f64(t);
            if (lane == 0) s_part[warp * PER + r] = t;
        }
        __syncthreads();
        if (warp == 0) {
            const double part = s_part[lane];
            if (parts) parts[sg * 32 + uint64_t(lane)] = part;
            const double total = __shfl_sync(0xffffffffu, lane_prefix(part, lane), 31);
            if (lane == 0) mass[sg] = total;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ uint64_t upper_index(const double *cdf, uint64_t n, double tau)
{
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (cdf[mid] <= tau) lo = mid + 1;
        else hi = mid;
    }
    return lo >= n ? n - 1 : lo;
}

__global__ void __launch_bounds__(kThreads) count_kernel(const double *__restrict__ segcdf, uint64_t nseg,
                                                         uint64_t stream_seed, uint64_t shots,
                                                         unsigned long long *__restrict__ counts)
{
    const double total = segcdf[nseg - 1];
    for (uint64_t base = uint64_t(blockIdx.x) * kThreads; base < shots; base += uint64_t(gridDim.x) * kThreads) {
        const uint64_t idx = base + threadIdx.x;
        const bool live = idx < shots && total > 0.0;
        uint64_t seg = ~0ULL;
        if (live) {
            const double u = uniform_open01(stream_seed ^ (kSeedShot + idx));
            seg = upper_index(segcdf, nseg, u * total);
        }
        // one atomic per distinct segment in the warp
        const unsigned peers = __match_any_sync(0xffffffffu, seg);
        const int leader = __ffs(peers) - 1;
        if (live && int(threadIdx.x & 31) == leader) atomicAdd(&counts[seg], static_cast<unsigned long long>(__popc(peers)));
    }
}

// exclusive scan of counts: block sums, scan of block sums, block scans
// Scan of n values in blocks of kScanBlock: per-block sums, one small scan over
// them, then each block's scan plus its offset. T = unsigned long long for the
// shot counts (exclusive offsets), double for the segment masses (inclusive CDF,
// written over the masses).
template <typename T>
__global__ void __launch_bounds__(kThreads) block_sum_kernel(const T *__restrict__ v, uint64_t n, T *__restrict__ bsum)
{
    __shared__ T sh[kThreads / 32];
    const uint64_t b0 = uint64_t(blockIdx.x) * kScanBlock;
    T acc = 0;
    for (uint64_t i = b0 + threadIdx.x; i < (n < b0 + kScanBlock ? n : b0 + kScanBlock); i += kThreads) acc += v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        T t = 0;
        for (int w = 0; w < kThreads / 32; w++) t += sh[w];
        bsum[blockIdx.x] = t;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) scan_small_kernel(T *v, uint64_t n)
{
    // one CTA, exclusive; n is at most a few thousand block sums. One thread adds them in
    // order, from shared memory: reading them one by one from global memory cost a round
    // trip to L2 each (19 us for the 64 of a 30-qubit state)
    __shared__ T sh[kThreads];
    __shared__ T s_run;
    if (threadIdx.x == 0) s_run = 0;
    for (uint64_t b = 0; b < n; b += kThreads) {
        if (b + threadIdx.x < n) sh[threadIdx.x] = v[b + threadIdx.x];
        __syncthreads();
        if (threadIdx.x == 0) {
            T run = s_run;
            for (uint32_t i = 0; i < kThreads && b + i < n; i++) {
                const T x = sh[i];
                sh[i] = run;
                run += x;
            }
            s_run = run;
        }
        __syncthreads();
        if (b + threadIdx.x < n) v[b + threadIdx.x] = sh[threadIdx.x];
        __syncthreads();
    }
}

// in and out may be the same array (every thread reads its own values first)
template <typename T, bool INCL>
__global__ void __launch_bounds__(kThreads) block_scan_kernel(const T *in, uint64_t n, const T *__restrict__ boff,
                                                              T *out)
{
    constexpr int PER = kScanBlock / kThreads;  // 16 consecutive values per thread
    __shared__ T sh[kThreads];
    const uint64_t b0 = uint64_t(blockIdx.x) * kScanBlock + uint64_t(threadIdx.x) * PER;
    T loc[PER];
    T acc = 0;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        loc[k] = (b0 + k < n) ? in[b0 + k] : T(0);
        acc += loc[k];
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 1; o < kThreads; o <<= 1) {
        const T x = threadIdx.x >= unsigned(o) ? sh[threadIdx.x - o] : T(0);
        __syncthreads();
        sh[threadIdx.x] += x;
        __syncthreads();
    }
    T run = boff[blockIdx.x] + (sh[threadIdx.x] - acc);
#pragma unroll
    for (int k = 0; k < PER; k++) {
        if (INCL) run += loc[k];
        if (b0 + k < n) out[b0 + k] = run;
        if (!INCL) run += loc[k];
    }
}

// Segment CDF, shot counts and offsets in one CTA, where the segments fit one scan block
// and the shots are few (a 20-qubit, 1024-shot draw spent 30 us in the seven launches
// this replaces). The CDF is scanned as block_scan_kernel does, so the draws are the same.
constexpr uint64_t kSmallShots = 16384;  // 64 searches a thread: about the launches' time

__global__ void __launch_bounds__(kThreads) small_draw_kernel(const double *mass, uint32_t nseg,
                                                              uint64_t stream_seed, uint32_t shots,
                                                              unsigned long long *__restrict__ counts,
                                                              unsigned long long *__restrict__ offsets,
                                                              uint32_t *heavy_count)
{
    constexpr int PER = kScanBlock / kThreads;
    __shared__ double cdf[kScanBlock];
    __shared__ __align__(8) uint32_t hits[kScanBlock];
    const uint32_t tid = threadIdx.x;
    chain_trigger();
    chain_wait();
    if (tid == 0) *heavy_count = 0;
    for (uint32_t i = tid; i < kScanBlock; i += kThreads) cdf[i] = i < nseg ? mass[i] : 0.0;
    __syncthreads();
    {
        double *sh = reinterpret_cast<double *>(hits);  // not counting yet
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < PER; k++) acc += cdf[tid * PER + k];
        sh[tid] = acc;
        __syncthreads();
        for (int o = 1; o < kThreads; o <<= 1) {
            const double x = tid >= unsigned(o) ? sh[tid - o] : 0.0;
            __syncthreads();
            sh[tid] += x;
            __syncthreads();
        }
        double run = 0.0 + (sh[tid] - acc);
#pragma unroll
        for (int k = 0; k < PER; k++) {
            run += cdf[tid * PER + k];
            cdf[tid * PER + k] = run;
        }
        __syncthreads();
        for (uint32_t i = tid; i < kScanBlock; i += kThreads) hits[i] = 0;
        __syncthreads();
    }
    const double total = cdf[nseg - 1];
    if (total > 0.0)
        for (uint32_t i = tid; i < shots; i += kThreads) {
            const double u = uniform_open01(stream_seed ^ (kSeedShot + uint64_t(i)));
            atomicAdd(&hits[upper_index(cdf, nseg, u * total)], 1u);
        }
    __syncthreads();
    uint32_t acc = 0;
#pragma unroll
    for (int k = 0; k < PER; k++) acc += hits[tid * PER + k];
    uint32_t *sh = reinterpret_cast<uint32_t *>(cdf);  // the searches are done
    sh[tid] = acc;
    __syncthreads();
    for (int o = 1; o < kThreads; o <<= 1) {
        const uint32_t x = tid >= unsigned(o) ? sh[tid - o] : 0u;
        __syncthreads();
        sh[tid] += x;
        __syncthreads();
    }
    uint32_t run = sh[tid] - acc;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const uint32_t i = tid * PER + k;
        if (i < nseg) {
            counts[i] = hits[i];
            offsets[i] = run;
        }
        run += hits[i];
    }
}

// Segments hit by at most kWarpMax shots. Warp w takes segments w, w + W, w + 2 W, ... (W
// warps in all): neighbouring segments of a state tend to have like masses, and a warp with 28
// of them in a row held up the others (10^6 shots from an uneven product state of 29 qubits).
// Registers are capped so that 4 CTAs fit an SM in complex64.
template <typename E>
__global__ void __launch_bounds__(kThreads, sizeof(E) == 8 ? 4 : 3) resolve_warp_kernel(const E *__restrict__ state, uint64_t nseg,
                                                                uint32_t seglen, const unsigned long long *counts,
                                                                const unsigned long long *offsets, uint64_t stream2,
                                                                uint64_t *__restrict__ real_out,
                                                                uint32_t *heavy_list, uint32_t *heavy_count,
                                                                const double *parts)
{
    chain_trigger();
    chain_wait();
    const int lane = threadIdx.x & 31;
    const uint64_t gwarp = (uint64_t(blockIdx.x) * kThreads + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * kThreads) >> 5;
    const uint32_t per_lane = (seglen + 31) / 32;  // amplitudes owned by a lane
    for (uint64_t g0 = gwarp; g0 < nseg; g0 += nwarps * 32) {
        const uint64_t gl = g0 + uint64_t(lane) * nwarps;
        const unsigned long long cl = gl < nseg ? counts[gl] : 0ULL;
        unsigned todo = __ballot_sync(0xffffffffu, cl != 0);
        if (cl > kWarpMax) heavy_list[atomicAdd(heavy_count, 1u)] = uint32_t(gl);
        todo &= __ballot_sync(0xffffffffu, cl <= kWarpMax);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint64_t g = g0 + uint64_t(src) * nwarps;
            const unsigned long long cnt = __shfl_sync(0xffffffffu, cl, src);
            const unsigned long long off = offsets[g];
            const E *seg = state + g * seglen;
            // lane range [lane*per_lane, (lane+1)*per_lane): its mass from the
            // segment kernel when kept, else read again
            const uint32_t lo = min(seglen, uint32_t(lane) * per_lane);
            const uint32_t hi = min(seglen, lo + per_lane);
            const double part = parts ? parts[g * 32 + uint64_t(lane)]
                                      : seglen == 4096 ? lane_range_mass(seg, lane) : range_mass(seg, lo, hi);
            const double incl = lane_prefix(part, lane);
            const double total = __shfl_sync(0xffffffffu, incl, 31);
            const double excl = incl - part;
            // this lane's shot
            double tau = 0.0;
            uint64_t mine = 0;  // its outcome
            if (uint64_t(lane) < cnt) tau = uniform_open01(stream2 ^ (kSeedOffset + off + uint64_t(lane))) * total;
            if (seglen == 4096) {
                // full segments: the owner range is 128 amplitudes, 4 per lane; they
                // are loaded at once and kept in registers, and the next shot's are
                // on their way while this shot is placed (the sums run in the same
                // order as the general path below, so the draws are the same)
                E cur[4], nxt[4];
                double t = __shfl_sync(0xffffffffu, tau, 0);
                int owner = __popc(__ballot_sync(0xffffffffu, incl <= t));
                if (owner < 32) {
#pragma unroll
                    for (int i = 0; i < 4; i++) cur[i] = __ldg(seg + uint32_t(owner) * 128u + uint32_t(lane) * 4u + i);
                }
#pragma unroll 1
                for (int j = 0; j < int(cnt); j++) {
                    double tn = 0.0;
                    int on = 32;
                    if (j + 1 < int(cnt)) {
                        tn = __shfl_sync(0xffffffffu, tau, j + 1);
                        on = __popc(__ballot_sync(0xffffffffu, incl <= tn));
                        if (on < 32) {
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                nxt[i] = __ldg(seg + uint32_t(on) * 128u + uint32_t(lane) * 4u + i);
                        }
                    }
                    uint64_t hit = seglen - 1;
                    if (owner < 32) {
                        const double obase = __shfl_sync(0xffffffffu, excl, owner);
                        double p[4], sp = 0.0;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            p[i] = prob(cur[i]);
                            sp += p[i];
                        }
                        double sincl = sp;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const double v = __shfl_up_sync(0xffffffffu, sincl, o);
                            if (lane >= o) sincl += v;
                        }
                        const int sl = __popc(__ballot_sync(0xffffffffu, obase + sincl <= t));
                        uint32_t found = 4;  // past this lane's sub-range
                        if (sl < 32 && lane == sl) {
                            double run = obase + sincl - sp;
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                run += p[i];
                                if (found == 4 && run > t) found = uint32_t(i);
                            }
                        }
                        const uint32_t fs = __shfl_sync(0xffffffffu, found, sl < 32 ? sl : 0);
                        hit = uint64_t(owner) * 128u + (sl < 32 ? uint32_t(sl) * 4u + fs : 128u);
                        if (hit >= seglen) hit = seglen - 1;
                    }
                    if (lane == j) mine = g * seglen + hit;
                    t = tn;
                    owner = on;
#pragma unroll
                    for (int i = 0; i < 4; i++) cur[i] = nxt[i];
                }
            } else for (int j = 0; j < int(cnt); j++) {
                const double t = __shfl_sync(0xffffffffu, tau, j);
                // owner lane: first lane whose inclusive prefix exceeds t
                const unsigned le = __ballot_sync(0xffffffffu, incl <= t);
                int owner = __popc(le);
                uint64_t hit;
                if (owner >= 32) {
                    hit = seglen - 1;
                } else {
                    // cooperative search in the owner's range: each lane takes a sub-range
                    const double obase = __shfl_sync(0xffffffffu, excl, owner);
                    const uint32_t olo = uint32_t(owner) * per_lane;
                    const uint32_t ohi = min(seglen, olo + per_lane);
                    const uint32_t sub = (per_lane + 31) / 32;
                    const uint32_t slo = min(ohi, olo + uint32_t(lane) * sub);
                    const uint32_t shi = min(ohi, slo + sub);
                    double sp = 0.0;
                    for (uint32_t k = slo; k < shi; k++) sp += prob(seg[k]);
                    double sincl = sp;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const double v = __shfl_up_sync(0xffffffffu, sincl, o);
                        if (lane >= o) sincl += v;
                    }
                    const unsigned le2 = __ballot_sync(0xffffffffu, obase + sincl <= t);
                    const int sl = __popc(le2);
                    uint32_t found = ohi;  // none below the end of the owner's range
                    if (sl < 32 && lane == sl) {
                        double run = obase + sincl - sp;
                        found = shi;
                        for (uint32_t k = slo; k < shi; k++) {
                            run += prob(seg[k]);
                            if (run > t) {
                                found = k;
                                break;
                            }
                        }
                    }
                    const uint32_t fs = __shfl_sync(0xffffffffu, found, sl < 32 ? sl : 0);
                    hit = (sl < 32) ? fs : ohi;
                    if (hit >= seglen) hit = seglen - 1;
                }
                if (lane == j) mine = g * seglen + hit;
            }
            if (uint64_t(lane) < cnt) real_out[off + uint64_t(lane)] = mine;
        }
    }
}

// Shared CDF of a heavy segment: entry k at k + k / 16, so the 16 consecutive
// entries a thread scans sit in distinct banks across the warp.
__device__ __forceinline__ uint32_t cdf_slot(uint32_t k) { return k + (k >> 4); }

__device__ __forceinline__ uint64_t upper_index_padded(const double *cdf, uint64_t n, double tau)
{
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (cdf[cdf_slot(uint32_t(mid))] <= tau) lo = mid + 1;
        else hi = mid;
    }
    return lo >= n ? n - 1 : lo;
}

template <typename E>
__global__ void __launch_bounds__(kThreads) resolve_cta_kernel(const E *__restrict__ state, uint32_t seglen,
                                                               const unsigned long long *counts,
                                                               const unsigned long long *offsets, uint64_t stream2,
                                                               uint64_t *__restrict__ real_out,
                                                               const uint32_t *heavy_list,
                                                               const uint32_t *heavy_count)
{
    extern __shared__ double cdf[];  // cdf_slot(seglen) entries
    __shared__ double s_warp[kThreads / 32];
    chain_trigger();
    chain_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nh = *heavy_count;
    // heavy segment h goes to CTA h mod grid, which places all of its shots
    for (uint32_t h = blockIdx.x; h < nh; h += gridDim.x) {
        const uint64_t g = heavy_list[h];
        const unsigned long long cnt = counts[g], off = offsets[g];
        // build the segment CDF once for all of its shots: coalesced loads, a serial
        // scan of each thread's consecutive range, a block scan of the range totals
        const E *seg = state + g * seglen;
        const uint32_t per = (seglen + kThreads - 1) / kThreads;
        const uint32_t lo = min(seglen, threadIdx.x * per), hi = min(seglen, lo + per);
        for (uint32_t k = threadIdx.x; k < seglen; k += kThreads) cdf[cdf_slot(k)] = prob(__ldg(seg + k));
        __syncthreads();
        double run = 0.0;
        for (uint32_t k = lo; k < hi; k++) {
            run += cdf[cdf_slot(k)];
            cdf[cdf_slot(k)] = run;
        }
        double incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        double add = incl - run;
        for (int w = 0; w < warp; w++) add += s_warp[w];
        for (uint32_t k = lo; k < hi; k++) cdf[cdf_slot(k)] += add;
        __syncthreads();
        const double total = cdf[cdf_slot(seglen - 1)];
        for (uint64_t j = threadIdx.x; j < cnt; j += kThreads) {
            const double tau = uniform_open01(stream2 ^ (kSeedOffset + off + j)) * total;
            real_out[off + j] = g * seglen + upper_index_padded(cdf, seglen, tau);
        }
        __syncthreads();  // cdf and s_warp are reused by the next heavy segment
    }
}

// Virtual words from byte tables (XORs of the map's columns), built by each CTA from the
// columns in the kernel's parameters.
struct MapTab {
    uint64_t t[8][256];
    uint64_t b;
    // all threads of the CTA; ends with a barrier
    __device__ __forceinline__ void build(const PermCols &c)
    {
        if (threadIdx.x == 0) b = c.b;
        for (uint32_t i = threadIdx.x; i < 256; i += kThreads)
            for (int k = 0; 8 * k < c.m; k++) {
                uint64_t v = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) v ^= ((i >> j) & 1u) ? c.col[8 * k + j] : 0ULL;
                t[k][i] = v;
            }
        m = c.m;
        __syncthreads();
    }
    __device__ __forceinline__ uint64_t word(uint64_t r) const
    {
        uint64_t v = b;
        for (int k = 0; 8 * k < m; k++) v ^= t[k][(r >> (8 * k)) & 255];
        return v;
    }
    int m;
};

__global__ void __launch_bounds__(kThreads) map_kernel(const uint64_t *real, uint64_t shots,
                                                       const __grid_constant__ PermCols cols,
                                                       uint64_t *__restrict__ words)
{
    __shared__ MapTab tab;
    tab.build(cols);
    chain_wait();
    for (uint64_t i = uint64_t(blockIdx.x) * kThreads + threadIdx.x; i < shots; i += uint64_t(gridDim.x) * kThreads)
        words[i] = tab.word(real[i]);
}

// ---------------------------------------------------------------------------
// Counts: the distinct outcomes of a draw and how often each came up, without
// copying the shots to the host. The draw leaves every shot's real index grouped
// by segment (segments in increasing order), so counting is per segment: a
// segment with at most kWarpMax shots sorts its offsets in one warp (bitonic
// network over the lanes) and run-length encodes them; a heavier segment (the
// sampler's heavy list) builds a histogram of its 2^12 offsets in shared memory.
// Pass 1 writes each segment's number of distinct outcomes, a scan of those gives
// every segment's first output slot, and pass 2 repeats the work and writes the
// (virtual word, count) pairs there, in increasing real index.

__device__ __forceinline__ uint32_t warp_sort32(uint32_t v, int lane)
{
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, v, j);
            const bool up = (lane & k) == 0;
            const bool low = (lane & j) == 0;
            v = (low == up) ? min(v, o) : max(v, o);
        }
    return v;
}

template <bool WRITE>
__global__ void __launch_bounds__(kThreads) count_light_kernel(const uint64_t *__restrict__ real, uint64_t nseg,
                                                               uint32_t seglen, const unsigned long long *counts,
                                                               const unsigned long long *offsets,
                                                               unsigned long long *nuniq,
                                                               const unsigned long long *uoff,
                                                               const __grid_constant__ PermCols cols,
                                                               uint64_t *__restrict__ words,
                                                               uint64_t *__restrict__ hits)
{
    [[maybe_unused]] __shared__ MapTab tab;
    if constexpr (WRITE) tab.build(cols);
    const int lane = threadIdx.x & 31;
    const uint64_t gwarp = (uint64_t(blockIdx.x) * kThreads + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * kThreads) >> 5;
    for (uint64_t g0 = gwarp * 32; g0 < nseg; g0 += nwarps * 32) {
        const uint64_t gl = g0 + uint64_t(lane);
        const unsigned long long cl = gl < nseg ? counts[gl] : 0ULL;
        if (!WRITE && gl < nseg && cl == 0) nuniq[gl] = 0;
        unsigned todo = __ballot_sync(0xffffffffu, cl != 0 && cl <= kWarpMax);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint64_t g = g0 + uint64_t(src);
            const uint32_t cnt = uint32_t(__shfl_sync(0xffffffffu, cl, src));
            const uint64_t base = g * seglen;
            const unsigned long long off = offsets[g];
            uint32_t key = 0xffffffffu;  // padding sorts last
            if (uint32_t(lane) < cnt) key = uint32_t(real[off + uint64_t(lane)] - base);
            key = warp_sort32(key, lane);
            const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
            const bool first = uint32_t(lane) < cnt && (lane == 0 || key != prev);
            const unsigned starts = __ballot_sync(0xffffffffu, first);
            if constexpr (!WRITE) {
                if (lane == 0) nuniq[g] = __popc(starts);
            } else if (first) {
                const unsigned above = starts & ~((2u << lane) - 1u);  // lane 31: 2u << 31 wraps to 0, nothing above
                const uint32_t next = above ? uint32_t(__ffs(above) - 1) : cnt;
                const uint64_t slot = uoff[g] + uint64_t(__popc(starts & ((1u << lane) - 1u)));
                words[slot] = tab.word(base + key);
                hits[slot] = next - uint32_t(lane);
            }
        }
    }
}

// heavy segment h goes to CTA h mod grid (shared histogram of seglen bins)
template <bool WRITE>
__global__ void __launch_bounds__(kThreads) count_heavy_kernel(const uint64_t *__restrict__ real, uint32_t seglen,
                                                               const unsigned long long *counts,
                                                               const unsigned long long *offsets,
                                                               const uint32_t *heavy_list,
                                                               const uint32_t *heavy_count,
                                                               unsigned long long *nuniq,
                                                               const unsigned long long *uoff,
                                                               const __grid_constant__ PermCols cols,
                                                               uint64_t *__restrict__ words,
                                                               uint64_t *__restrict__ hits)
{
    __shared__ uint32_t hist[4096];
    __shared__ uint32_t s_warp[kThreads / 32];
    [[maybe_unused]] __shared__ MapTab tab;
    if constexpr (WRITE) tab.build(cols);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nh = *heavy_count;
    const uint32_t per = (seglen + kThreads - 1) / kThreads;  // bins of a thread (16 for full segments)
    for (uint32_t h = blockIdx.x; h < nh; h += gridDim.x) {
        const uint64_t g = heavy_list[h];
        const unsigned long long cnt = counts[g], off = offsets[g];
        const uint64_t base = g * seglen;
        for (uint32_t k = threadIdx.x; k < seglen; k += kThreads) hist[k] = 0;
        __syncthreads();
        for (uint64_t j = threadIdx.x; j < cnt; j += kThreads) atomicAdd(&hist[uint32_t(real[off + j] - base)], 1u);
        __syncthreads();
        const uint32_t lo = min(seglen, uint32_t(threadIdx.x) * per), hi = min(seglen, lo + per);
        uint32_t mine = 0;
        for (uint32_t k = lo; k < hi; k++) mine += hist[k] != 0;
        // block exclusive scan of the per-thread distinct counts
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (int w = 0; w < kThreads / 32; w++) {
            before += w < warp ? s_warp[w] : 0;
            total += s_warp[w];
        }
        if constexpr (!WRITE) {
            if (threadIdx.x == 0) nuniq[g] = total;
        } else {
            uint64_t slot = uoff[g] + before + incl - mine;
            for (uint32_t k = lo; k < hi; k++)
                if (hist[k]) {
                    words[slot] = tab.word(base + k);
                    hits[slot] = hist[k];
                    slot++;
                }
        }
        __syncthreads();  // hist and s_warp are reused by the next heavy segment
    }
}

__global__ void count_total_kernel(const unsigned long long *nuniq, const unsigned long long *uoff, uint64_t nseg,
                                   unsigned long long *total)
{
    *total = uoff[nseg - 1] + nuniq[nseg - 1];
}

}  // namespace

cudaError_t run_counts(const SamplerScratch &sc, int m, const PermCols &cols, unsigned long long *nuniq,
                       unsigned long long *uoff, unsigned long long *total, uint64_t *words, uint64_t *hits,
                       int pass, int sms, cudaStream_t st, uint64_t &kernels)
{
    const uint64_t local = 1ULL << m;
    const uint32_t seglen = uint32_t(std::min<uint64_t>(4096, local));
    const uint64_t nseg = local / seglen;
    const uint64_t nblk = (nseg + kScanBlock - 1) / kScanBlock;
    const uint64_t warps_needed = (nseg + 31) / 32;
    const unsigned gw = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((warps_needed * 32 + kThreads - 1) / kThreads,
                                                                          uint64_t(sms) * 8)));
    const unsigned gh = unsigned(sms) * 4;
    if (pass == 1) {
        count_light_kernel<false><<<gw, kThreads, 0, st>>>(sc.real, nseg, seglen, sc.counts, sc.offsets, nuniq,
                                                           nullptr, cols, nullptr, nullptr);
        count_heavy_kernel<false><<<gh, kThreads, 0, st>>>(sc.real, seglen, sc.counts, sc.offsets, sc.heavy_list,
                                                           sc.heavy_count, nuniq, nullptr, cols, nullptr,
                                                           nullptr);
        block_sum_kernel<unsigned long long><<<unsigned(nblk), kThreads, 0, st>>>(nuniq, nseg, sc.bsum);
        scan_small_kernel<unsigned long long><<<1, kThreads, 0, st>>>(sc.bsum, nblk);
        block_scan_kernel<unsigned long long, false><<<unsigned(nblk), kThreads, 0, st>>>(nuniq, nseg, sc.bsum, uoff);
        count_total_kernel<<<1, 1, 0, st>>>(nuniq, uoff, nseg, total);
        kernels += 6;
    } else {
        count_light_kernel<true><<<gw, kThreads, 0, st>>>(sc.real, nseg, seglen, sc.counts, sc.offsets, nuniq, uoff,
                                                          cols, words, hits);
        count_heavy_kernel<true><<<gh, kThreads, 0, st>>>(sc.real, seglen, sc.counts, sc.offsets, sc.heavy_list,
                                                          sc.heavy_count, nuniq, uoff, cols, words, hits);
        kernels += 2;
    }
    return cudaGetLastError();
}

// One layout routine serves both the size query and the carving, so the two can
// never disagree.
static size_t layout(SamplerScratch *sc, uint8_t *base, uint64_t nseg, uint64_t shots, bool with_parts)
{
    const uint64_t nblk = (nseg + kScanBlock - 1) / kScanBlock;
    size_t b = 0;
    auto take = [&](size_t x) {
        uint8_t *p = base ? base + b : nullptr;
        b += (x + 255) & ~size_t(255);
        return p;
    };
    uint8_t *segcdf = take(nseg * 8);
    uint8_t *heavy_count = take(16);
    uint8_t *counts = take(nseg * 8);
    uint8_t *offsets = take(nseg * 8);
    uint8_t *bsum = take(nblk * 8);
    uint8_t *heavy = take(nseg * 4);
    uint8_t *real = take(shots * 8);
    uint8_t *words = take(shots * 8);
    uint8_t *parts = with_parts ? take(nseg * 32 * 8) : nullptr;
    if (sc) {
        sc->parts = reinterpret_cast<double *>(parts);
        sc->segcdf = reinterpret_cast<double *>(segcdf);
        sc->heavy_count = reinterpret_cast<uint32_t *>(heavy_count);
        sc->counts = reinterpret_cast<unsigned long long *>(counts);
        sc->offsets = reinterpret_cast<unsigned long long *>(offsets);
        sc->bsum = reinterpret_cast<unsigned long long *>(bsum);
        sc->heavy_list = reinterpret_cast<uint32_t *>(heavy);
        sc->real = reinterpret_cast<uint64_t *>(real);
        sc->words = reinterpret_cast<uint64_t *>(words);
    }
    return b;
}

size_t SamplerScratch::need_bytes(uint64_t nseg, uint64_t shots, bool parts)
{
    return layout(nullptr, nullptr, nseg, shots, parts);
}

void SamplerScratch::carve(uint8_t *base, uint64_t nseg, uint64_t shots, bool parts)
{
    layout(this, base, nseg, shots, parts);
}

namespace {

template <typename E>
cudaError_t draw(const E *state, int m, uint64_t shots, uint64_t stream_seed, uint64_t *real_out, const PermCols &cols,
                 uint64_t *words, SamplerScratch &sc, int sms, cudaStream_t st, uint64_t &kernels)
{
    const uint64_t local = 1ULL << m;
    const uint32_t seglen = uint32_t(std::min<uint64_t>(4096, local));
    const uint64_t nseg = local / seglen;
    const uint64_t nblk = (nseg + kScanBlock - 1) / kScanBlock;
    const uint64_t stream2 = mix_seed_host(stream_seed, 1);
    const uint64_t slots = uint64_t(sms) * 8;  // CTAs at most
    auto grid = [&](uint64_t ctas) { return unsigned(std::max<uint64_t>(1, std::min(ctas, slots))); };
    // a CTA per segment while that leaves no more CTAs than fit
    if (seglen == 4096 && nseg <= slots)
        seg_mass_cta_kernel<E><<<grid(nseg), kThreads, 0, st>>>(state, nseg, sc.segcdf, sc.parts);
    else
        seg_mass_kernel<E><<<grid((nseg * 32 + kThreads - 1) / kThreads), kThreads, 0, st>>>(state, nseg, seglen, sc.segcdf,
                                                                                          sc.parts);
    kernels++;
    // Only a small draw's launches are chained (chain.cuh): in a large one the next kernel's
    // waiting CTAs take room from the one that runs (10^6 shots at 27 qubits 0.54 instead of 0.49 ms).
    const bool small = nblk == 1 && shots <= kSmallShots;
    if (small) {
        const cudaError_t e = launch_chained(true, small_draw_kernel, 1, kThreads, 0, st, sc.segcdf, nseg, stream_seed,
                                             shots, sc.counts, sc.offsets, sc.heavy_count);
        if (e != cudaSuccess) return e;
        kernels++;
    } else {
        cudaError_t e = cudaMemsetAsync(sc.heavy_count, 0, sizeof(uint32_t), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(sc.counts, 0, nseg * 8, st);
        if (e != cudaSuccess) return e;
        double *bsum_d = reinterpret_cast<double *>(sc.bsum);  // the counts' scan reuses it afterwards
        block_sum_kernel<double><<<unsigned(nblk), kThreads, 0, st>>>(sc.segcdf, nseg, bsum_d);
        scan_small_kernel<double><<<1, kThreads, 0, st>>>(bsum_d, nblk);
        block_scan_kernel<double, true><<<unsigned(nblk), kThreads, 0, st>>>(sc.segcdf, nseg, bsum_d, sc.segcdf);
        count_kernel<<<grid((shots + kThreads - 1) / kThreads), kThreads, 0, st>>>(sc.segcdf, nseg, stream_seed, shots,
                                                                                 sc.counts);
        block_sum_kernel<unsigned long long><<<unsigned(nblk), kThreads, 0, st>>>(sc.counts, nseg, sc.bsum);
        scan_small_kernel<unsigned long long><<<1, kThreads, 0, st>>>(sc.bsum, nblk);
        block_scan_kernel<unsigned long long, false><<<unsigned(nblk), kThreads, 0, st>>>(sc.counts, nseg, sc.bsum,
                                                                                         sc.offsets);
        kernels += 7;
    }
    // a warp per segment, as many warps as fit on the chip (4 CTAs an SM); 32 segments queued
    // on each warp left a 20-qubit state's 256 to 8 warps (120 us)
    const uint64_t ctas = std::min<uint64_t>((nseg * 32 + kThreads - 1) / kThreads, uint64_t(sms) * 4);
    cudaError_t e = launch_chained(small, resolve_warp_kernel<E>, grid(ctas), kThreads, 0, st, state, nseg, seglen, sc.counts,
                                   sc.offsets, stream2, real_out, sc.heavy_list, sc.heavy_count, sc.parts);
    kernels++;
    if (e == cudaSuccess && shots > kWarpMax) {  // fewer cannot make a segment heavy
        const size_t smem = size_t(seglen + seglen / 16 + 1) * 8;
        e = launch_chained(small, resolve_cta_kernel<E>, grid(std::min<uint64_t>(nseg, uint64_t(sms) * 2)), kThreads, smem, st,
                           state, seglen, sc.counts, sc.offsets, stream2, real_out, sc.heavy_list, sc.heavy_count);
        kernels++;
    }
    if (e == cudaSuccess && words) {
        e = launch_chained(small, map_kernel, grid((shots + kThreads - 1) / kThreads), kThreads, 0, st, real_out, shots, cols,
                           words);
        kernels++;
    }
    return e;
}

}  // namespace

cudaError_t run_sampler(const void *state, int elem_bytes, int m, uint64_t shots, uint64_t stream_seed,
                        const PermCols &cols, uint64_t *real_out, uint64_t *words, SamplerScratch &sc, int sms,
                        cudaStream_t st, uint64_t &kernels)
{
    if (elem_bytes == 8)
        return draw(static_cast<const float2 *>(state), m, shots, stream_seed, real_out, cols, words, sc, sms, st, kernels);
    return draw(static_cast<const double2 *>(state), m, shots, stream_seed, real_out, cols, words, sc, sms, st, kernels);
}

uint64_t mix_seed_host(uint64_t base, uint64_t salt)
{
    // mix_seed, measure_cuda.cu:103-109
    uint64_t z = base + 0x9e3779b97f4a7c15ULL + salt;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

}  // namespace zxh
