// Host check of the batched engines' programs (rq_plan.cuh): symmetric_program (QAOA on the kept half
// of a state with psi(x) = psi(~x)) and packed_program (real states, two amplitudes an element).  Every
// program is run the way the kernels run it -- tiles, register slots, thread bits, op order -- in
// double precision and compared with the circuit on the whole state; every tile must cover each index
// once and every phase each tile offset once.
#include <complex>
#include <cstdio>
#include <random>

#include "rq_plan.cuh"

using namespace rqp;
using C = std::complex<double>;

static int fails = 0;
#define CHECK(c, ...)                       \
    do {                                    \
        if (!(c)) {                         \
            ++fails;                        \
            std::printf(__VA_ARGS__);       \
            std::printf("\n");              \
        }                                   \
    } while (0)

// runs the sweeps; op(regs, ph, o, U) applies one op to a thread's registers
template <class F>
static void run_program(const std::vector<SweepDesc>& descs, const std::vector<PhaseDesc>& phases,
                        const std::vector<SwOp>& ops, uint32_t rb, uint32_t epv, std::vector<C>& st, F op) {
    for (const auto& d : descs) {
        const uint32_t T = 1u << (d.m - rb), VPT = (1u << rb) / epv, M = 1u << d.m;
        std::vector<char> seen(st.size(), 0);
        for (uint64_t tile = 0; tile < st.size() >> d.m; ++tile) {
            uint64_t base = 0;
            for (uint32_t b = 0; b < d.nonlocal_count; ++b)
                if ((tile >> b) & 1) base |= 1ull << d.nonlocal[b];
            std::vector<C> sm(M);
            std::vector<uint64_t> at(M);
            for (uint32_t tid = 0; tid < T; ++tid) {
                const uint64_t x = (uint64_t)tid * epv;
                uint64_t dep = x & ((1ull << d.c) - 1);
                for (uint32_t b = d.c; b < d.m; ++b)
                    if ((x >> b) & 1) dep |= 1ull << d.local_global[b];
                for (uint32_t j = 0; j < VPT; ++j)
                    for (uint32_t k = 0; k < epv; ++k) {
                        const uint64_t g = ((base ^ d.gj[j]) | dep) + k;
                        const uint32_t e = j * T * epv + tid * epv + k;
                        CHECK(g < st.size() && !seen[g], "index %llu twice or out of range", (unsigned long long)g);
                        if (g >= st.size()) return;
                        seen[g] = 1;
                        sm[e] = st[g];
                        at[e] = g;
                    }
            }
            for (uint32_t p = d.phase_begin; p < d.phase_end; ++p) {
                const PhaseDesc& ph = phases[p];
                std::vector<char> hit(M, 0);
                CHECK(ph.nt == d.m - rb, "thread bits");
                for (uint32_t tid = 0; tid < T; ++tid) {
                    uint32_t eb = 0;
                    uint64_t U = base;
                    for (uint32_t b = 0; b < ph.nt; ++b)
                        if ((tid >> b) & 1) {
                            eb |= 1u << ph.tbit_local[b];
                            U |= 1ull << ph.tbit_global[b];
                        }
                    if (U >> SELECTOR) U = (U ^ d.selmask) & ~(1ull << SELECTOR);
                    CHECK(at[eb] == U, "thread index %llu, tile holds %llu", (unsigned long long)U, (unsigned long long)at[eb]);
                    std::vector<C> reg(1u << rb);
                    for (uint32_t i = 0; i < reg.size(); ++i) {
                        const uint32_t a = eb ^ ph.lut[i];
                        CHECK(a < M && !hit[a], "offset %u twice", a);
                        hit[a] = 1;
                        CHECK(ph.slut[i] == swz_host(ph.lut[i], epv == 2 ? 4 : 3), "slut");
                        reg[i] = sm[a];
                    }
                    for (uint32_t o = ph.op_begin; o < ph.op_end; ++o) op(reg, ph, ops[o], U);
                    for (uint32_t i = 0; i < reg.size(); ++i) sm[eb ^ ph.lut[i]] = reg[i];
                }
            }
            for (uint32_t e = 0; e < M; ++e) st[at[e]] = sm[e];
        }
        for (char s : seen) CHECK(s, "index missed");
    }
}

static void check_symmetric(uint32_t n, uint32_t m, uint32_t rb, uint32_t epv, uint32_t p, std::mt19937& r) {
    std::uniform_real_distribution<double> u(-1.5, 1.5);
    std::vector<std::pair<uint32_t, uint32_t>> edges;
    for (uint32_t a = 0; a < n; ++a)
        for (uint32_t b = a + 1; b < n; ++b)
            if (u(r) > 0.6) edges.push_back({a, b});
    std::vector<uint64_t> nb(32, 0);
    for (auto& e : edges) nb[e.first] |= 1ull << e.second, nb[e.second] |= 1ull << e.first;
    std::vector<double> ga(p), be(p);
    std::vector<PGate> g;
    for (uint32_t l = 0; l < p; ++l) {
        ga[l] = u(r), be[l] = u(r);
        PGate ph{};
        ph.type = OP_CPH;
        ph.param = (uint16_t)l;
        ph.span = (1ull << n) - 1;
        g.push_back(ph);
        for (uint32_t q = 0; q < n; ++q) {
            PGate x{};
            x.type = OP_RXP;
            x.q0 = q;
            x.param = (uint16_t)l;
            g.push_back(x);
        }
    }
    auto cut = [&](uint64_t x) {
        int c = 0;
        for (auto& e : edges) c += ((x >> e.first) ^ (x >> e.second)) & 1;
        return c;
    };
    std::vector<C> full(1ull << n, std::ldexp(1.0, 0) / std::sqrt(std::ldexp(1.0, (int)n)));
    for (uint32_t l = 0; l < p; ++l) {
        for (uint64_t x = 0; x < full.size(); ++x) full[x] *= std::polar(1.0, -ga[l] * ((double)edges.size() - 2 * cut(x)));
        for (uint32_t q = 0; q < n; ++q)
            for (uint64_t x = 0; x < full.size(); ++x)
                if (!((x >> q) & 1)) {
                    C a = full[x], b = full[x | (1ull << q)];
                    const C is(0, std::sin(be[l]));
                    full[x] = std::cos(be[l]) * a - is * b;
                    full[x | (1ull << q)] = std::cos(be[l]) * b - is * a;
                }
    }
    std::vector<SweepDesc> descs;
    std::vector<PhaseDesc> phases;
    std::vector<SwOp> ops;
    symmetric_program(g, n, std::min(n - 1, m), rb, epv, descs, phases, ops);
    std::vector<C> st(1ull << (n - 1), std::sqrt(std::ldexp(1.0, -(int)n)));
    run_program(descs, phases, ops, rb, epv, st, [&](std::vector<C>& reg, const PhaseDesc& ph, const SwOp& o, uint64_t U) {
        if (o.type == OP_RXP) {
            CHECK(o.k0 >= 0, "Rx without a slot");
            for (uint32_t i = 0; i < reg.size(); ++i)
                if (!((i >> o.k0) & 1)) {
                    C a = reg[i], b = reg[i | (1u << o.k0)];
                    const C is(0, std::sin(be[o.param]));
                    reg[i] = std::cos(be[o.param]) * a - is * b;
                    reg[i | (1u << o.k0)] = std::cos(be[o.param]) * b - is * a;
                }
        } else {   // as cut_plan_nb / cut_nb: counts from the slots' neighbour masks
            int c0 = 0;
            for (uint32_t v = 0; v < 32; ++v)
                if ((U >> v) & 1) c0 += __builtin_popcountll(nb[v] & ~U);
            for (uint32_t i = 0; i < reg.size(); ++i) {
                int c = c0;
                for (uint32_t s = 0; s < rb; ++s)
                    if ((i >> s) & 1) {
                        const uint64_t ns = nb[ph.slot_global[s]];
                        c += __builtin_popcountll(ns) - 2 * __builtin_popcountll(ns & U);
                        for (uint32_t t = s + 1; t < rb; ++t)
                            if (((i >> t) & 1) && ((ns >> ph.slot_global[t]) & 1)) c -= 2;
                    }
                reg[i] *= std::polar(1.0, -ga[o.param] * ((double)edges.size() - 2 * c));
            }
        }
    });
    double err = 0;
    for (uint64_t x = 0; x < full.size(); ++x) err = std::max(err, std::abs(full[x] - st[x < st.size() ? x : ~x & (full.size() - 1)]));
    CHECK(err < 1e-12, "symmetric n=%u m=%u rb=%u: %g", n, m, rb, err);
}

static void check_packed(uint32_t n, uint32_t mloc, uint32_t rb, uint32_t epv, uint32_t depth, bool reverse, std::mt19937& r) {
    std::uniform_real_distribution<double> u(-3, 3);
    std::vector<double> th(n * depth);
    for (auto& t : th) t = u(r);
    std::vector<PGate> g;
    for (uint32_t l = 0; l < depth; ++l) {
        for (uint32_t q = 0; q < n; ++q) {
            PGate y{};
            y.type = OP_RYP;
            y.q0 = q;
            y.param = (uint16_t)(l * n + q);
            g.push_back(y);
        }
        for (uint32_t q = 0; q + 1 < n; ++q) {
            PGate z{};
            z.type = OP_CZ;
            z.q0 = q;
            z.q1 = q + 1;
            g.push_back(z);
        }
    }
    if (reverse) std::reverse(g.begin(), g.end());
    std::vector<double> full(1ull << n, 0.0);
    for (auto& x : full) x = u(r);
    const std::vector<double> start = full;
    for (auto& o : g)
        for (uint64_t x = 0; x < full.size(); ++x) {
            if (o.type == OP_CZ) {
                if (((x >> o.q0) & 1) && ((x >> o.q1) & 1)) full[x] = -full[x];
            } else if (!((x >> o.q0) & 1)) {
                const double c = std::cos(th[o.param] / 2), s = std::sin(th[o.param] / 2);
                const double a = full[x], b = full[x | (1ull << o.q0)];
                full[x] = c * a - s * b;
                full[x | (1ull << o.q0)] = s * a + c * b;
            }
        }
    std::vector<SweepDesc> descs;
    std::vector<PhaseDesc> phases;
    std::vector<SwOp> ops;
    packed_program(g, n, mloc, std::min(n - 1, mloc), rb, epv, descs, phases, ops);
    std::vector<C> st(1ull << (n - 1));
    for (uint64_t j = 0; j < st.size(); ++j) st[j] = C(start[2 * j], start[2 * j + 1]);
    run_program(descs, phases, ops, rb, epv, st, [&](std::vector<C>& reg, const PhaseDesc& ph, const SwOp& o, uint64_t U) {
        const double c = std::cos(th[o.param] / 2), s = std::sin(th[o.param] / 2);
        for (uint32_t i = 0; i < reg.size(); ++i) {
            const int b0 = o.k0 >= 0 ? (i >> o.k0) & 1 : (U >> o.q0) & 1;
            if (o.type == OP_CZL) {
                uint64_t x = U;
                for (uint32_t s = 0; s < rb; ++s)
                    if ((i >> s) & 1) x |= 1ull << ph.slot_global[s];
                if (__builtin_popcountll(x & (x >> 1) & o.mat) & 1) reg[i] = -reg[i];
            } else if (o.type == OP_RY0) {
                reg[i] = C(c * reg[i].real() - s * reg[i].imag(), s * reg[i].real() + c * reg[i].imag());
            } else if (o.type == OP_CZ0) {
                if (b0) reg[i] = std::conj(reg[i]);
            } else {
                CHECK(o.k0 >= 0, "Ry without a slot");
                if (!((i >> o.k0) & 1)) {
                    const C a = reg[i], b = reg[i | (1u << o.k0)];
                    reg[i] = c * a - s * b;
                    reg[i | (1u << o.k0)] = s * a + c * b;
                }
            }
        }
    });
    double err = 0;
    for (uint64_t j = 0; j < st.size(); ++j) err = std::max(err, std::abs(st[j] - C(full[2 * j], full[2 * j + 1])));
    CHECK(err < 1e-11, "packed n=%u m=%u rb=%u: %g", n, mloc, rb, err);
}

int main() {
    std::mt19937 r(5);
    int count = 0;
    for (uint32_t epv = 1; epv <= 2; ++epv)
        for (uint32_t rb = 3; rb <= 5; ++rb)
            for (uint32_t n = rb + 2; n <= 13; ++n)
                for (uint32_t m = rb + 2; m <= 9; ++m) {
                    if (m < 6 && n > m) continue;   // a tile holds the five contiguous qubits and at least one more
                    check_symmetric(n, m, rb, epv, 1 + n % 3, r);
                    check_packed(n, m, rb, epv, 1 + n % 4, (n + m) & 1, r);
                    count += 2;
                }
    std::printf("%d programs, %d failures\n", count, fails);
    return fails != 0;
}
