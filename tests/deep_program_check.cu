// Host check of deep batched programs: no sweep has more phases than its shared memory holds, and an
// ansatz whose single tile is cut for that still equals the circuit (the checks of batch_program_check.cu).
#define main batch_program_check_main
#include "batch_program_check.cu"
#undef main

static size_t most_phases(uint32_t n, uint32_t depth, uint32_t mloc, uint32_t rb, uint32_t epv, size_t* sweeps) {
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
    std::vector<SweepDesc> descs;
    std::vector<PhaseDesc> phases;
    std::vector<SwOp> ops;
    const uint32_t m = std::min(n - 1, mloc);
    packed_program(g, n, mloc, m, rb, epv, descs, phases, ops);
    size_t most = 0;
    for (const auto& d : descs) {
        most = std::max<size_t>(most, d.phase_end - d.phase_begin);
        // as the launch asks for it: the tile, the descriptors and 2 KB of static shared memory
        const size_t bytes = ((size_t)(16 / epv) << m) + (d.phase_end - d.phase_begin) * sizeof(PhaseDesc) + 2048;
        CHECK(bytes <= 227 * 1024, "n=%u depth=%u epv=%u: a sweep of %u phases needs %zu bytes", n, depth, epv,
              d.phase_end - d.phase_begin, bytes);
    }
    *sweeps = descs.size();
    return most;
}

int main() {
    std::mt19937 r(7);
    size_t a = 0, b = 0;
    for (uint32_t n : {7u, 13u, 14u, 15u})
        for (uint32_t depth : {1u, 560u, 700u}) {
            most_phases(n, depth, 13, 5, 2, &a);
            most_phases(n, depth, 12, 4, 1, &b);
        }
    most_phases(14, 1400, 13, 5, 2, &a);
    // QAOA takes at most 64 layers: never near the limit
    for (uint32_t n = 7; n <= 18; ++n)
        for (uint32_t epv = 1; epv <= 2; ++epv) {
            std::vector<PGate> g;
            for (uint32_t l = 0; l < 64; ++l) {
                PGate ph{};
                ph.type = OP_CPH;
                ph.span = (1ull << n) - 1;
                g.push_back(ph);
                for (uint32_t q = 0; q < n; ++q) {
                    PGate x{};
                    x.type = OP_RXP;
                    x.q0 = q;
                    g.push_back(x);
                }
            }
            std::vector<SweepDesc> d;
            std::vector<PhaseDesc> p;
            std::vector<SwOp> o;
            const uint32_t m = std::min(n - 1, epv == 2 ? 13u : 12u);
            symmetric_program(g, n, m, epv == 2 ? 5 : 4, epv, d, p, o);
            for (const auto& s : d) CHECK(s.phase_end - s.phase_begin <= sweep_phase_limit(m, epv) / 2, "QAOA of %u", n);
        }
    // a state of one tile stays one sweep while it fits
    most_phases(14, 560, 13, 5, 2, &a);
    most_phases(13, 400, 12, 4, 1, &b);
    CHECK(a == 1 && b == 1, "%zu and %zu sweeps", a, b);
    most_phases(14, 600, 13, 5, 2, &a);
    most_phases(13, 450, 12, 4, 1, &b);
    CHECK(a == 2 && b == 2, "%zu and %zu sweeps past the limit", a, b);
    check_packed(14, 13, 5, 2, 580, false, r);
    check_packed(13, 12, 4, 1, 430, true, r);
    std::printf("%d failures\n", fails);
    return fails != 0;
}
