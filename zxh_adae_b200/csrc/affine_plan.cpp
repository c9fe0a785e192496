// affine_plan.cpp -- host side of the affine tile pass (affine.cu): the tile's basis, the
// selectors in tile coordinates and the windows' entries.
#include "affine.h"
#include "host.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace zxh {

namespace {

int top_bit(uint64_t x) { return 63 - __builtin_clzll(x); }

uint64_t reduced(uint64_t v, const std::vector<uint64_t> &ech)
{
    for (uint64_t b : ech)
        if ((v >> top_bit(b)) & 1) v ^= b;
    return v;
}

void insert(uint64_t v, std::vector<uint64_t> &ech)
{
    ech.push_back(v);
    std::sort(ech.rbegin(), ech.rend());
}

}  // namespace

int AffBuild::Room::add(uint64_t delta)
{
    uint64_t v = delta;  // delta modulo the high deltas, their parts' leading bits cleared
    for (const High &h : high)
        if ((v >> (kAffRun + top_bit(h.part))) & 1) v ^= h.delta;
    if (v >> kAffRun) {
        if (high.size() >= size_t(kAffHigh)) return -1;
        high.push_back({v >> kAffRun, v});
        std::sort(high.begin(), high.end(), [](const High &x, const High &y) { return x.part > y.part; });
        return 1;
    }
    if (low.size() >= size_t(kAffRun)) return -1;
    v = reduced(v, low);
    if (!v) return -1;
    insert(v, low);
    return 0;
}

bool AffBuild::init(int eb, int mm, const std::vector<U3Op> &gates, const std::vector<uint64_t> &deltas, bool adjoint_matrix,
                    const std::vector<uint32_t> *gen, const std::vector<uint32_t> *slot)
{
    elem_bytes = eb;
    m = mm;
    std::memset(&dev, 0, sizeof(dev));
    for (int d = 0; d < 2; d++) {
        entries[d].clear();
        terms[d].clear();
    }
    form = 2;
    dev.scale = 1.0;
    // What a matrix may miss its form by, but for what is known to be real. Nothing in
    // complex128: a phase of 1e-15 dropped from every gate of a deep circuit adds up. In
    // complex64 the amplitudes round at 6e-8.
    const double round = elem_bytes == 8 ? 1e-15 : 0.0;
    if (m < kAffBits || m > kAffMaxBits) return false;
    dev.m = uint32_t(m);
    Room room;
    int nlow = 0, nhigh = 0;
    std::vector<int> at;
    for (const U3Op &g : gates) {
        if (g.has_ctrl || !g.delta) return false;
        const int kind = room.add(g.delta);
        if (kind < 0) return false;
        at.push_back(kind ? kAffRun + nhigh++ : nlow++);
        dev.basis[at.back()] = g.delta;
    }
    // The run's other basis vectors are single bits, moved by the low gates' deltas so that
    // no selector of those gates sees them.
    for (int b = 0; b < kAffRun && nlow < kAffRun; b++) {
        const uint64_t r = reduced(1ULL << b, room.low);
        if (!r) continue;
        insert(r, room.low);
        uint64_t v = 1ULL << b;
        for (size_t i = 0; i < gates.size(); i++)
            if (at[i] < kAffRun && parity64(gates[i].sel.alpha & (1ULL << b))) v ^= gates[i].delta;
        dev.basis[nlow++] = v;
    }
    // The other high coordinates are deltas of other qubits (lowest first: long runs), which
    // no other qubit's selector sees; so every selector of the map has one high coordinate
    // at most.
    std::vector<uint64_t> others(deltas);
    std::sort(others.begin(), others.end());
    for (uint64_t d : others) {
        if (nhigh == kAffHigh) break;
        if (room.add(d) == 1) dev.basis[kAffRun + nhigh++] = d;
    }
    if (nlow != kAffRun || nhigh != kAffHigh) return false;
    uint64_t piv = low_mask(kAffRun);
    for (const Room::High &h : room.high) piv |= 1ULL << (top_bit(h.part) + kAffRun);
    int t = 0;
    for (int b = 0; b < m; b++)
        if (!((piv >> b) & 1)) dev.tr[t++] = 1ULL << b;
    dev.ntiles = 1ULL << t;

    for (size_t i = 0; i < gates.size(); i++) {
        const U3Op &g = gates[i];
        const int s = selector(g.sel);
        if (s < 0) return false;
        // the gate's selector flips with its own coordinate and no other of its kind
        for (int k = 0; k < kAffBits; k++) {
            const bool sees = parity64(g.sel.alpha & dev.basis[k]);
            if (k == at[i] ? !sees : sees && (k >= kAffRun || at[i] < kAffRun)) return false;
        }
        AffGateDev &d = dev.gate[at[i]];
        cd w[4] = {g.u[0], g.u[1], g.u[2], g.u[3]};
        if (adjoint_matrix) {  // U^dagger
            w[0] = std::conj(g.u[0]);
            w[1] = std::conj(g.u[2]);
            w[2] = std::conj(g.u[1]);
            w[3] = std::conj(g.u[3]);
        }
        if (g.real)
            for (cd &x : w) x = x.real();
        for (int q = 0; q < 4; q++) {
            d.u[2 * q] = w[q].real();
            d.u[2 * q + 1] = w[q].imag();
            if (!(std::fabs(w[q].imag()) <= round)) form = 0;
        }
        d.sel = uint32_t(s);
        d.gen = gen ? (*gen)[i] : 0u;
        d.slot = slot ? (*slot)[i] : 0u;
        dev.gates |= 1u << at[i];
        const double c = w[0].real(), sn = w[2].real();
        const bool rot = std::fabs(c - w[3].real()) <= round && std::fabs(sn + w[1].real()) <= round;
        const bool refl = std::fabs(c + w[3].real()) <= round && std::fabs(sn - w[1].real()) <= round;
        // an X generator's gradient (RX by a multiple of 2 pi is real) takes the general form
        if (d.gen == 2 || !(rot || refl)) form = std::min(form, 1);
        const bool mu = std::fabs(c) < std::fabs(sn);
        if (mu) dev.mu |= 1u << at[i];
        if (!rot) dev.refl |= 1u << at[i];
        // from the other member of a pair the factor changes sign: a rotation's s, a reflection's c
        if (mu == rot) (at[i] < kAffRun ? dev.neg_low : dev.neg_high) |= 1ULL << s;
        d.rot = mu ? c / sn : sn / c;
        dev.scale *= mu ? sn : c;
    }
    // the order gates are applied in: layouts A, C, B
    double before = 1.0;
    for (int k : {4, 5, 6, 7, 0, 1, 2, 3, 8, 9, 10, 11}) {
        AffGateDev &d = dev.gate[k];
        d.gscale = before;
        if (!((dev.gates >> k) & 1)) continue;
        const double f = ((dev.mu >> k) & 1) ? d.u[4] : d.u[0];
        before *= f * f;
    }
    return true;
}

int AffBuild::selector(const Sel &s)
{
    const uint64_t a = s.alpha & low_mask(m);
    for (uint32_t i = 0; i < dev.nsel; i++)
        if (dev.alpha[i] == a && int((dev.lw[0] >> i) & 1) == s.beta) return int(i);
    if (dev.nsel >= uint32_t(kAffMaxSel)) return -1;
    int k = -1;
    for (int j = 0; j < kAffHigh; j++)
        if (parity64(a & dev.basis[kAffRun + j])) {
            if (k >= 0) return -1;
            k = j;
        }
    const uint32_t i = dev.nsel++;
    dev.alpha[i] = a;
    coord_[i] = k;
    for (uint32_t l = 0; l < (1u << kAffRun); l++) {
        uint64_t v = 0;
        for (int b = 0; b < kAffRun; b++)
            if ((l >> b) & 1) v ^= dev.basis[b];
        dev.lw[l] |= uint64_t(parity64(a & v) ^ s.beta) << i;
    }
    return int(i);
}

bool AffBuild::add_window(int which, const std::vector<DiagTerm> &w, const std::vector<uint32_t> *gk,
                          const std::vector<uint32_t> *slot, bool inverse)
{
    if (w.size() > size_t(kAffMaxTerms)) return false;
    const AffDev saved = dev;
    std::vector<AffEntryDev> none, of[kAffHigh];
    std::vector<AffTermDev> ts;
    uint32_t pairs = 0;
    for (size_t i = 0; i < w.size(); i++) {
        const DiagTerm &t = w[i];
        int s0 = selector(t.s0), s1 = t.two ? selector(t.s1) : 0xff;
        if (s0 < 0 || s1 < 0) {
            dev = saved;
            return false;
        }
        if (s0 == s1) s1 = 0xff;  // S and S = S
        int k0 = coord_[s0], k1 = s1 == 0xff ? -1 : coord_[s1];
        if (s1 != 0xff && k1 >= 0 && (k0 < 0 || k1 < k0)) {
            std::swap(s0, s1);
            std::swap(k0, k1);
        }
        AffEntryDev e;
        std::memset(&e, 0, sizeof(e));
        e.s0 = uint8_t(s0);
        e.s1 = uint8_t(s1);
        e.coef = phase_turns(inverse ? -t.theta : t.theta);
        AffTermDev g;
        std::memset(&g, 0, sizeof(g));
        g.s0 = uint8_t(s0);
        g.s1 = uint8_t(s1);
        g.k0 = uint8_t(k0);
        g.k1 = uint8_t(k1);
        g.gk = gk ? uint8_t((*gk)[i]) : uint8_t(0);
        g.slot = slot ? (*slot)[i] : 0u;
        if (k0 < 0) {
            none.push_back(e);
        } else if (k1 < 0) {
            e.kind = s1 == 0xff ? 1 : 2;
            of[k0].push_back(e);
        } else if (k0 == k1) {
            e.kind = 5;
            of[k0].push_back(e);
        } else {
            e.kind = 3;
            e.pair = uint8_t(aff_pair(k0, k1));
            g.pair = e.pair;
            e.first = !((pairs >> e.pair) & 1);
            pairs |= 1u << e.pair;
            of[k0].push_back(e);
            std::swap(e.s0, e.s1);
            e.kind = 4;
            of[k1].push_back(e);
        }
        ts.push_back(g);
    }
    for (AffTermDev &g : ts)  // rows of the pair sums: the pairs in use, in order
        g.pair = uint8_t(__builtin_popcount(pairs & ((1u << g.pair) - 1u)));
    AffWinDev &d = dev.win[which];
    d.n0 = uint32_t(none.size());
    d.pairs = pairs;
    d.nterms = uint32_t(ts.size());
    std::vector<AffEntryDev> &out = entries[which];
    out = none;
    for (int k = 0; k < kAffHigh; k++) {
        d.ck[k] = uint32_t(out.size());
        out.insert(out.end(), of[k].begin(), of[k].end());
    }
    d.ck[kAffHigh] = uint32_t(out.size());
    terms[which] = ts;
    return true;
}

}  // namespace zxh
