// rq_pauli_plan.cuh -- which kernel of rq_reduce.cu sums which Pauli string (host code): strings without
// X in passes of k_pauli_z, the others in passes of k_pauli_span, whose X patterns span eight dimensions.
#pragma once

#include "rq_internal.cuh"

#include <algorithm>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

namespace rqs {

constexpr uint32_t SMALL_QUBITS = 13;   // states of k_pauli_small
constexpr int SK = 16, STB = 9;         // strings of a pass of k_pauli_span; a tile index is STB thread bits, then register bits
struct SpanString {
    uint64_t z;
    uint16_t lx, lz;     // X and sign masks on the tile's local bits
    uint8_t mode, odd;   // mode: register bit held at 0, or the number of register bits: walk all
    uint16_t pad;
};
struct SpanPass {
    uint64_t basis[8];   // bits above the run
    uint8_t free_bit[24];   // the other bits above the run, low to high: the tile number's bits
    uint32_t k, row0;       // its strings, and the row of the first
    SpanString s[SK];
};

inline double re_ipow(uint32_t k) {
    switch (k & 3u) {
        case 0: return 1.0;
        case 2: return -1.0;
        default: return 0.0;
    }
}

struct PauliPlan {
    bool small = false;
    std::vector<uint32_t> zs;             // strings of k_pauli_z in row order
    std::vector<SpanPass> spans;
    uint32_t rows = 0;                    // one per string
    uint32_t zblocks = 0, sblocks = 0, stride = 0;
    std::vector<uint32_t> row_of;         // string -> row
    std::vector<double> factor;           // string -> factor of its sum
    const rq::PauliMask* terms = nullptr;
};

// The strings not yet in a pass, in order, and per X pattern (of the bits above the run) the queue of its
// strings: a pass with a full basis finds the strings of its 256 patterns by lookups instead of a walk over
// all that are left, which is quadratic: 100,000 unrelated strings of 24 qubits take 0.09 s to plan, seconds by a walk.
class StringQueue {
  public:
    // terms[ids[0..count)] with x = xmask & mask
    StringQueue(const rq::PauliMask* terms, std::vector<uint32_t> ids, uint64_t mask)
        : terms_(terms), ids_(std::move(ids)), mask_(mask), left_(ids_.size()), taken_(ids_.size(), 0) {
        if (left_ <= FEW) return;
        group_.resize(left_);
        next_.assign(left_, NONE);
        uint32_t bits = 10;
        while ((1ull << bits) < 4 * left_) ++bits;
        shift_ = 64 - bits;
        table_.assign((size_t)1 << bits, NONE);
        std::vector<uint32_t> last;
        for (uint32_t k = 0; k < left_; ++k) {
            const uint64_t x = pattern(k);
            uint32_t& slot = table_[find(x)];
            if (slot == NONE) {
                slot = (uint32_t)x_.size();
                x_.push_back(x);
                head_.push_back(k);
                last.push_back(k);
            } else {
                next_[last[slot]] = k;
                last[slot] = k;
            }
            group_[k] = slot;
        }
    }
    bool empty() const { return left_ == 0; }
    uint64_t pattern(uint32_t k) const { return terms_[ids_[k]].xmask & mask_; }

    // The next pass, at most SK strings: in order until the basis is full(), every pattern that reduced()
    // leaves something of joining it by add(); then, in order, those whose pattern the basis spans.
    template <class Reduce, class Add, class Full>
    std::vector<uint32_t> take(Reduce reduced, Add add, Full full, const uint64_t* basis) {
        std::vector<uint32_t> out;
        while (first_ < ids_.size() && taken_[first_]) ++first_;
        uint32_t k = first_;
        for (; k < ids_.size() && out.size() < (size_t)SK && !full(); ++k) {
            if (taken_[k]) continue;
            if (const uint64_t r = reduced(pattern(k))) add(r);
            pop(k, out);
        }
        if (out.size() == (size_t)SK || left_ == 0) return out;
        if (table_.empty()) {
            for (; k < ids_.size() && out.size() < (size_t)SK; ++k)
                if (!taken_[k] && reduced(pattern(k)) == 0) pop(k, out);
            return out;
        }
        std::priority_queue<uint32_t, std::vector<uint32_t>, std::greater<uint32_t>> heads;
        uint64_t x = 0;
        for (uint32_t u = 0; u < 256; ++u) {   // Gray code over the span
            if (u) x ^= basis[__builtin_ctz(u)];
            const uint32_t g = table_[find(x)];
            if (g != NONE && head_[g] != NONE) heads.push(head_[g]);
        }
        while (!heads.empty() && out.size() < (size_t)SK) {
            const uint32_t h = heads.top();
            heads.pop();
            pop(h, out);
            if (next_[h] != NONE) heads.push(next_[h]);
        }
        return out;
    }

  private:
    static constexpr uint32_t NONE = ~0u;
    static constexpr size_t FEW = 8192;   // a walk over so few is as fast as the lookups
    size_t find(uint64_t x) const {      // slot of x, or the empty one where it would go
        size_t i = (x * 0x9E3779B97F4A7C15ull) >> shift_;
        while (table_[i] != NONE && x_[table_[i]] != x) i = (i + 1) & (table_.size() - 1);
        return i;
    }
    void pop(uint32_t k, std::vector<uint32_t>& out) {   // k is the first of its pattern that is left
        taken_[k] = 1;
        --left_;
        if (!table_.empty()) head_[group_[k]] = next_[k];
        out.push_back(ids_[k]);
    }
    const rq::PauliMask* terms_;
    std::vector<uint32_t> ids_;
    uint64_t mask_;
    size_t left_;
    std::vector<char> taken_;
    uint32_t first_ = 0, shift_ = 0;
    std::vector<uint32_t> group_, next_, table_, head_;
    std::vector<uint64_t> x_;
};

inline void plan_strings(uint32_t n, int32_t prec, int sms, const rq::PauliMask* terms, uint32_t nterms, PauliPlan& P) {
    P.terms = terms;
    P.rows = nterms;
    P.row_of.assign(nterms, 0);
    P.factor.resize(nterms);
    for (uint32_t k = 0; k < nterms; ++k) {
        const rq::PauliMask& t = terms[k];
        const bool odd = __builtin_popcountll(t.xmask & t.pmask) & 1;
        P.factor[k] = t.xmask == 0 ? re_ipow(t.ny) : 2.0 * re_ipow(odd ? t.ny + 1 : t.ny);
    }
    if (n <= SMALL_QUBITS) {
        P.small = true;
        for (uint32_t k = 0; k < nterms; ++k) P.row_of[k] = k;
        return;
    }
    std::vector<uint32_t> ids;
    for (uint32_t k = 0; k < nterms; ++k) {
        if (terms[k].xmask == 0) {
            P.row_of[k] = (uint32_t)P.zs.size();
            P.zs.push_back(k);
        } else {
            ids.push_back(k);
        }
    }
    uint32_t row = (uint32_t)P.zs.size();
    const uint32_t C = prec == RQ_F32 ? 5 : 4, RB = prec == RQ_F32 ? 4 : 3;
    const uint64_t low = (1ull << C) - 1;
    StringQueue left(terms, std::move(ids), ~low);
    while (!left.empty()) {
        SpanPass sp{};
        sp.row0 = row;
        uint64_t pivot[8];
        uint32_t dim = 0;
        auto reduced = [&](uint64_t x) {
            for (uint32_t b = 0; b < dim; ++b)
                if (x & pivot[b]) x ^= sp.basis[b];
            return x;
        };
        auto add = [&](uint64_t v) {   // v reduced and not zero: clear its pivot from the others
            const uint64_t pv = 1ull << (63 - __builtin_clzll(v));
            for (uint32_t b = 0; b < dim; ++b)
                if (sp.basis[b] & pv) sp.basis[b] ^= v;
            pivot[dim] = pv;
            sp.basis[dim++] = v;
        };
        const std::vector<uint32_t> take = left.take(reduced, add, [&] { return dim == 8; }, sp.basis);
        for (uint32_t q = C; dim < 8; ++q)
            if (const uint64_t r = reduced(1ull << q)) add(r);
        uint64_t pivots = 0;
        for (uint32_t b = 0; b < 8; ++b) pivots |= pivot[b];
        uint32_t nf = 0;
        for (uint32_t q = C; q < n; ++q)
            if (!((pivots >> q) & 1)) sp.free_bit[nf++] = (uint8_t)q;
        for (uint32_t k : take) {
            const rq::PauliMask& t = terms[k];
            SpanString& ss = sp.s[sp.k];
            uint32_t lx = (uint32_t)(t.xmask & low), lz = (uint32_t)(t.pmask & low);
            for (uint32_t b = 0; b < 8; ++b) {
                if (t.xmask & pivot[b]) lx |= 1u << (C + b);
                if (__builtin_popcountll(sp.basis[b] & t.pmask) & 1) lz |= 1u << (C + b);
            }
            ss.z = t.pmask;
            ss.lx = (uint16_t)lx;
            ss.lz = (uint16_t)lz;
            ss.odd = (uint8_t)(__builtin_popcountll(t.xmask & t.pmask) & 1);
            const uint32_t xr = lx >> STB;
            ss.mode = (uint8_t)(xr ? 31 - __builtin_clz(xr) : RB);
            if (!xr) P.factor[k] *= 0.5;   // walked from both ends
            P.row_of[k] = row++;
            ++sp.k;
        }
        P.spans.push_back(sp);
    }
    P.zblocks = P.zs.empty() ? 0 : (uint32_t)std::min<uint64_t>(1ull << (n - 12), (uint64_t)sms * 2);
    P.sblocks = P.spans.empty() ? 0 : (uint32_t)std::min<uint64_t>(1ull << (n - C - 8), (uint64_t)sms);
    P.stride = std::max(P.zblocks, P.sblocks);
}

}  // namespace rqs
