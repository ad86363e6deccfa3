// Batches as the server admits them: what they take stays within the budget —
// test code (tests/test_server_budget.py).
#include "../libfastlib_b200/csrc/wah_budget.h"
#include <cmath>
#include <random>
#include <vector>
using namespace wah;
extern "C" int budget_model(uint32_t seed, int rounds) {
    std::mt19937_64 r(seed);
    auto upto = [&](double most) { return (uint64_t)std::exp(std::uniform_real_distribution<>(0, std::log(most))(r)); };
    for (int i = 0; i < rounds; ++i) {
        const uint32_t nslots = 1 + r() % 16;
        const size_t budget = upto(8e9), kept = slot_kept(budget, nslots);
        if (kept * nslots > budget / 4) return 1;
        size_t taken = 0, in_use = 0;  // what the slots' batches take; what is charged
        for (uint32_t s = 0; s < nslots; ++s) {
            uint64_t items = 0, ids = 0;
            for (int k = 1 + (int)upto(1000); k > 0; --k) {
                const uint64_t t = upto(40000), cap = r() % 2 ? upto(1e6) : 0;
                if (in_use + request_charge(t, cap) > budget - nslots * kept) break;
                in_use += request_charge(t, cap);
                items += t;
                ids += cap;
            }
            taken += batch_scratch(items, kept) + 4 * ids;
        }
        if (taken > budget) return 2;
    }
    return 0;
}
