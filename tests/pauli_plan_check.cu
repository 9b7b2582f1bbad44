// Host check of the plan of Pauli strings (rq_pauli_plan.cuh): the same passes, rows and factors as a
// walk over all strings left gives, for every family, and a time that grows with the number of strings.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "rq_pauli_plan.cuh"

using namespace rqs;

// the passes as sets of strings, by definition: in order, a string whose X pattern is in the span of the
// pass's patterns or extends it to at most eight dimensions, until the pass has SK strings
static std::vector<std::vector<uint32_t>> passes_by_walk(const std::vector<rq::PauliMask>& t, uint64_t mask) {
    std::vector<uint32_t> left;
    for (uint32_t k = 0; k < t.size(); ++k)
        if (t[k].xmask) left.push_back(k);
    std::vector<std::vector<uint32_t>> out;
    while (!left.empty()) {
        std::vector<uint64_t> basis;   // by descending leading bit
        std::vector<uint32_t> take, rest;
        for (uint32_t k : left) {
            uint64_t x = t[k].xmask & mask;
            for (uint64_t b : basis) x = std::min(x, x ^ b);
            if (take.size() == (size_t)SK || (x && basis.size() == 8)) {
                rest.push_back(k);
                continue;
            }
            if (x) {
                basis.push_back(x);
                std::sort(basis.rbegin(), basis.rend());
            }
            take.push_back(k);
        }
        out.push_back(take);
        left.swap(rest);
    }
    return out;
}

int main() {
    std::mt19937_64 r(3);
    int fails = 0, plans = 0;
    for (uint32_t n : {14u, 16u, 24u, 33u})
        for (int32_t prec : {(int32_t)RQ_F32, (int32_t)RQ_F64})
            for (uint32_t count : {1u, 16u, 17u, 300u, 8192u, 8193u})
                for (int family = 0; family < 6; ++family) {
                    if (prec == RQ_F64 && n == 33) continue;
                    const uint64_t all = (1ull << n) - 1;
                    std::vector<rq::PauliMask> t(count);
                    for (uint32_t k = 0; k < count; ++k) {
                        t[k].pmask = r() & all;
                        t[k].ny = (uint32_t)(r() & 3);
                        switch (family) {
                            case 0: t[k].xmask = r() & all; break;                                  // unrelated
                            case 1: t[k].xmask = 1ull << (r() % n); break;                          // X fields
                            case 2: t[k].xmask = (r() % 5 + 1) << (n - 3); break;                   // few patterns
                            case 3: t[k].xmask = (1ull << (k % n)) ^ (1ull << ((k + 2) % n)); break;
                            case 4: t[k].xmask = (r() & r() & r()) & all; break;                    // sparse, some zero
                            default: t[k].xmask = r() % 3 ? (r() & 15) : 0x3Full << (n - 6); break;  // inside a run
                        }
                    }
                    PauliPlan P;
                    plan_strings(n, prec, 148, t.data(), count, P);
                    const auto want = passes_by_walk(t, ~((1ull << (prec == RQ_F32 ? 5 : 4)) - 1));
                    bool ok = P.spans.size() == want.size();
                    uint32_t row = (uint32_t)P.zs.size();
                    for (size_t p = 0; ok && p < want.size(); ++p) {
                        ok = P.spans[p].k == want[p].size() && P.spans[p].row0 == row;
                        for (size_t j = 0; ok && j < want[p].size(); ++j) {
                            ok = P.row_of[want[p][j]] == row + j && P.spans[p].s[j].z == t[want[p][j]].pmask;
                            // the pattern is the sum of the basis vectors that its local X mask names
                            const uint32_t C = prec == RQ_F32 ? 5 : 4;
                            uint64_t x = P.spans[p].s[j].lx & ((1u << C) - 1);
                            for (int b = 0; b < 8; ++b)
                                if ((P.spans[p].s[j].lx >> (C + b)) & 1) x ^= P.spans[p].basis[b];
                            ok = ok && x == t[want[p][j]].xmask;
                        }
                        row += (uint32_t)want[p].size();
                    }
                    ok = ok && row == count;
                    if (!ok) {
                        ++fails;
                        std::printf("n=%u prec=%d count=%u family=%d differs\n", n, prec, count, family);
                    }
                    ++plans;
                }
    // unrelated strings: a walk over all that are left took 3 to 6 s
    for (int family = 0; family < 2; ++family) {
        std::vector<rq::PauliMask> t(100000);
        for (auto& m : t) m = {family ? 1ull << (r() % 24) : 1 + r() % ((1ull << 24) - 1), r() & 0xFFFFFF, 0};
        PauliPlan P;
        const auto t0 = std::chrono::steady_clock::now();
        plan_strings(24, RQ_F32, 148, t.data(), (uint32_t)t.size(), P);
        const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        std::printf("100000 strings, family %d: %.4f s, %zu passes\n", family, s, P.spans.size());
        if (s > 1.0) ++fails;
    }
    std::printf("%d plans, %d failures\n", plans, fails);
    return fails != 0;
}
