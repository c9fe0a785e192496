// permute.h -- the state in virtual order (permute.cu): the launcher and the host
// plan of its tiles.
#pragma once

#include "core.h"

#include <cuda_runtime.h>

namespace zxh {

constexpr int kPermBits = 12;  // most tile bits

// out index of real address r: b ^ the XOR of col[j] over the set bits j of r.
struct PermCols {
    uint64_t col[64];
    uint64_t b;
    int m;
};

// A tile's entries, numbered in read order (bit i of the number: real vector rvec[i],
// shared-memory slot spos[i]) and in write order (bit i: output vector wimg[i], slot
// wpos[i]); tile bit j adds the real vector tr[j], whose image is ti[j].
struct PermDev {
    uint32_t d, pad;
    uint64_t ntiles, b;
    uint64_t rvec[kPermBits], wimg[kPermBits];
    uint32_t spos[kPermBits], wpos[kPermBits];
    uint64_t tr[64], ti[64];
};

// Plans tiles of at most dmax bits with runs of 2^cmax amplitudes on both sides; bank:
// log2 entries of a 128-byte shared-memory row. False if the columns are dependent.
bool perm_plan(const PermCols &cols, int cmax, int dmax, int bank, PermDev &p);

// out[b ^ B r] = (gre + i gim) * state[r] for every r < 2^m; the other entries of out
// are left alone.
cudaError_t run_permute(const void *state, const PermCols &cols, double gre, double gim, void *out, int elem_bytes,
                        int sms, cudaStream_t st);

}  // namespace zxh
