// affine.h -- the affine tile pass (affine.cu): its device records, the host builder and
// the launcher.
#pragma once

#include "core.h"

#include <cuda_runtime.h>

#include <vector>

namespace zxh {

constexpr int kAffBits = 12;      // tile coordinates
constexpr int kAffMaxBits = 32;   // largest state
constexpr int kAffRun = 4;        // coordinates 0..3 span the low 4 real bits
constexpr int kAffHigh = kAffBits - kAffRun;
constexpr int kAffPairs = kAffHigh * (kAffHigh - 1) / 2;
constexpr int kAffMaxSel = 64;
constexpr int kAffMaxTerms = 128;
constexpr int kAffMaxEntries = 2 * kAffMaxTerms;

// Index of the pair (i, j), i < j, of high coordinates.
__host__ __device__ constexpr int aff_pair(int i, int j) { return i * (2 * kAffHigh - i - 1) / 2 + (j - i - 1); }

// The gate on a coordinate: u00, u01, u10, u11 (re, im; U^dagger in adjoint passes), its
// qubit's selector, the gradient's generator (0 none, 1 Y, 2 X) and slot.
// Factored passes: one coefficient of a rotation [[c, -s], [s, c]] or a reflection [[c, s],
// [s, -c]] (bit of AffDev::refl) factored out, rot = s / c and factor c where |c| >= |s|, else
// (bit of AffDev::mu) rot = c / s and factor s; gscale is the square of the factors of the
// gates applied before it.
struct AffGateDev {
    double u[8];
    double rot, gscale;
    uint32_t sel, gen, slot, pad;
};

// One contribution of a window term to its phase polynomial over the high coordinates
// (bits y_k): selector s is y_k ^ f_s with its coordinate k, or f_s with none; f_s is fixed
// by the tile and the run position. kind 0: no coordinate; 1: s0 has one; 2: s0 has one,
// s1 none; 3: both have one (s0's is the lower); 4: the other half of kind 3, listed at
// s1's coordinate with the selectors swapped; 5: both have the same one.
struct AffEntryDev {
    uint8_t s0, s1, kind, pair;  // s1 = 0xff: one selector; pair: kind 3, aff_pair of the coordinates
    uint32_t first;              // kind 3: the first entry of its pair
    int64_t coef;                // 64-bit turns
};

// A window term of an adjoint pass (gradient kinds as in GrowTermDev): k0, k1 the high
// coordinates of its selectors or 0xff, pair the row of the pair sums it reads.
struct AffTermDev {
    uint8_t s0, s1, k0, k1;
    uint8_t gk, pair, pad[2];
    uint32_t slot, pad2;
};

// A window: entries [0, n0) of kind 0, those of high coordinate k at [ck[k], ck[k + 1]);
// pairs: bit aff_pair(i, j) where the polynomial has the product y_i y_j.
struct AffWinDev {
    uint32_t n0, ck[kAffHigh + 1], pairs, nterms;
    uint64_t off_entries, off_terms;
};

struct AffDev {
    uint32_t m, gates, nsel, pad;  // gates: bit k = coordinate k has one
    uint32_t mu, refl;             // factored passes: the gates with rot = c / s, the reflections
    double scale;                  // the product of the factors, negated by the parity of these
    uint64_t neg_high, neg_low;    // selector bits (high coordinates' gates: of the run position;
                                   // low ones': of the tile)
    uint64_t ntiles;
    uint64_t basis[kAffBits], tr[64];      // tile coordinates; real vectors of the tile bits
    uint64_t alpha[kAffMaxSel], lw[1 << kAffRun];  // selector masks; bit s of lw[l]: f_s of run position l
    AffGateDev gate[kAffBits];
    AffWinDev win[2];
};

// Builds one pass over commuting 2x2 gates on distinct qubits of a 2^m state whose map has
// the pair deltas `deltas` (one per qubit, every qubit of the map).
struct AffBuild {
    int elem_bytes = 8, m = 0;
    AffDev dev;
    std::vector<AffEntryDev> entries[2];
    std::vector<AffTermDev> terms[2];
    // 0: complex matrices; 1: every gate's is real; 2: every gate is a real rotation or reflection
    int form = 2;

    // The coordinates of a pass: up to 8 deltas independent modulo the run bits (high), up to 4
    // that are not but are independent of all others (low: inside the run bits, or the sum of
    // such a vector and of high deltas, as the gates of a CX fan-in have).
    struct Room {
        struct High { uint64_t part, delta; };  // part: delta >> kAffRun reduced by those before it
        std::vector<High> high;                 // echelon form, largest part first
        std::vector<uint64_t> low;              // echelon form of the low coordinates' run parts
        int add(uint64_t delta);  // 1: a high coordinate, 0: a low one, -1: no room (nothing changes)
    };
    bool init(int elem_bytes, int m, const std::vector<U3Op> &gates, const std::vector<uint64_t> &deltas,
              bool adjoint_matrix = false, const std::vector<uint32_t> *gen = nullptr,
              const std::vector<uint32_t> *slot = nullptr);
    // which: 0 before the gates, 1 after (adjoint passes: 0 is undone before the gates).
    // False where a selector flips with several coordinates or a table is full; nothing
    // changes then.
    bool add_window(int which, const std::vector<DiagTerm> &w, const std::vector<uint32_t> *gk = nullptr,
                    const std::vector<uint32_t> *slot = nullptr, bool inverse = false);

  private:
    int selector(const Sel &s);  // index, -1 if it does not fit
    int coord_[kAffMaxSel];      // high coordinate of a selector, -1 if none
};

// The pass at poff of the blob over psi (read from psi_src where given); lam != nullptr:
// the adjoint form, gradients added to grads[slot]. toff: the phase table (unused without
// windows). chained: directly after another kernel of the run (chain.cuh).
cudaError_t run_affine(const uint8_t *dblob, uint64_t poff, uint64_t toff, uint64_t ntiles, int elem_bytes, int form,
                       void *psi, const void *psi_src, void *lam, double *grads, bool chained, int sms, cudaStream_t st);

}  // namespace zxh
