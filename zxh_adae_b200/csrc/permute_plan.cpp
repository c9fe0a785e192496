// permute_plan.cpp -- host plan of the virtual-order pass (permute.cu): linear algebra
// over GF(2) on at most 64 vectors.
#include "permute.h"

#include <algorithm>
#include <vector>

namespace zxh {

namespace {

int top_bit(uint64_t x) { return 63 - __builtin_clzll(x); }

// A set of independent vectors in echelon form on a key.
struct Echelon {
    std::vector<uint64_t> key;
    // key reduced by the set; appended when it is independent
    bool add(uint64_t k)
    {
        for (uint64_t b : key) k = std::min(k, k ^ b);
        if (!k) return false;
        key.push_back(k);
        std::sort(key.rbegin(), key.rend());
        return true;
    }
};

}  // namespace

bool perm_plan(const PermCols &cols, int cmax, int dmax, int bank, PermDev &p)
{
    const int m = cols.m;
    auto image = [&](uint64_t r) {
        uint64_t v = 0;
        for (int j = 0; j < m; j++)
            if ((r >> j) & 1) v ^= cols.col[j];
        return v;
    };
    Echelon rank;
    for (int j = 0; j < m; j++)
        if (!rank.add(cols.col[j])) return false;
    const int c = std::min(cmax, m);

    // g: a basis of the real vectors whose image lies below 2^c, images in reduced
    // echelon form, smallest first
    struct Null { uint64_t img, r; };
    std::vector<Null> elim, g;
    for (int j = 0; j < m; j++) {
        Null v{cols.col[j], 1ULL << j};
        for (const Null &e : elim)
            if (((v.img >> c) ^ (e.img >> c)) < (v.img >> c)) {
                v.img ^= e.img;
                v.r ^= e.r;
            }
        if (v.img >> c) {
            elim.push_back(v);
            std::sort(elim.begin(), elim.end(), [](const Null &a, const Null &b) { return a.img > b.img; });
        } else {
            g.push_back(v);
        }
    }
    for (size_t i = 0; i < g.size(); i++) {
        size_t best = i;
        for (size_t k = i; k < g.size(); k++)
            if (g[k].img > g[best].img) best = k;
        std::swap(g[i], g[best]);
        const int t = top_bit(g[i].img);
        for (size_t k = 0; k < g.size(); k++)
            if (k != i && ((g[k].img >> t) & 1)) {
                g[k].img ^= g[i].img;
                g[k].r ^= g[i].r;
            }
    }
    std::sort(g.begin(), g.end(), [](const Null &a, const Null &b) { return a.img < b.img; });

    // read basis: e_0 .. e_{c-1}, then the high parts of g in reduced echelon form,
    // then single bits up to dmax
    std::vector<uint64_t> u;
    const uint64_t low = low_mask(c);
    auto reduce = [&](uint64_t v) {
        v &= ~low;
        for (uint64_t b : u)
            if ((v >> top_bit(b)) & 1) v ^= b;
        return v;
    };
    auto extend = [&](uint64_t v) {
        v = reduce(v);
        if (!v) return;
        const int t = top_bit(v);
        for (uint64_t &b : u)
            if ((b >> t) & 1) b ^= v;
        u.push_back(v);
    };
    for (const Null &v : g) extend(v.r);
    for (int j = c; j < m && c + int(u.size()) < dmax; j++) extend(1ULL << j);
    const int d = c + int(u.size());
    auto coords = [&](uint64_t v) {  // read number of a vector of the tile
        uint32_t q = uint32_t(v & low);
        for (size_t k = 0; k < u.size(); k++)
            if ((v >> top_bit(u[k])) & 1) q |= 1u << (c + k);
        return q;
    };
    std::vector<uint64_t> rb;
    for (int j = 0; j < c; j++) rb.push_back(1ULL << j);
    rb.insert(rb.end(), u.begin(), u.end());

    // write basis: g, completed by read vectors
    std::vector<uint64_t> wb;
    Echelon have;
    for (const Null &v : g) {
        have.add(coords(v.r));
        wb.push_back(v.r);
    }
    for (uint64_t v : rb)
        if (int(wb.size()) < d && have.add(coords(v))) wb.push_back(v);

    // shared-memory slots: the read number with its run bits below `bank` XORed by a
    // linear function of its high bits, searched so that the first 2^bank writes in
    // write order (one 128-byte row) fall on different banks
    std::vector<uint32_t> f(u.size(), 0), bestf = f;
    auto slot = [&](uint32_t q, const std::vector<uint32_t> &ff) {
        for (size_t k = 0; k < ff.size(); k++)
            if ((q >> (c + k)) & 1) q ^= ff[k];
        return q;
    };
    const int bb = std::min(bank, c);
    int best = -1;
    uint32_t rng = 12345;
    for (int tries = 0; tries < 64 && best < std::min(bb, int(wb.size())); tries++) {
        for (size_t k = 0; k < f.size(); k++) {
            rng = rng * 1664525u + 1013904223u;
            // first guess: the high bits in turn
            f[k] = tries == 0 ? 1u << (k % size_t(std::max(bb, 1))) : (rng >> 16) & ((1u << bb) - 1u);
        }
        Echelon banks;
        int r = 0;
        for (int k = 0; k < std::min(bb, int(wb.size())); k++)
            r += banks.add(slot(coords(wb[size_t(k)]), f) & ((1u << bb) - 1u));
        if (r > best) {
            best = r;
            bestf = f;
        }
    }

    p = PermDev();
    p.d = uint32_t(d);
    p.b = cols.b;
    for (int k = 0; k < d; k++) {
        p.rvec[k] = rb[size_t(k)];
        p.spos[k] = slot(1u << k, bestf);
        p.wimg[k] = image(wb[size_t(k)]);
        p.wpos[k] = slot(coords(wb[size_t(k)]), bestf);
    }
    uint64_t piv = low;
    for (uint64_t b : u) piv |= 1ULL << top_bit(b);
    int t = 0;
    for (int j = 0; j < m; j++)
        if (!((piv >> j) & 1)) {
            p.tr[t] = 1ULL << j;
            p.ti[t] = cols.col[j];
            t++;
        }
    p.ntiles = 1ULL << t;
    return true;
}

}  // namespace zxh
