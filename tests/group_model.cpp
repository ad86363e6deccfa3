// CPU model of the count-1 flags told from the words around one-group runs
// (single_flag and its walks, wah_core.cuh / wah_gop.cuh) — test code.
//
// Random operands are combined group by group, the runs' words taken from
// single_flag, and compared with the walk's step states (cpu_model.cpp's
// merge).  tests/test_group_model.py runs it.
#include "cpu_model.cpp"
#include <random>

namespace {
struct Str { V w; std::vector<uint32_t> st, cov; };  // words, their first groups, the word of every group
Str expand(const V& w) {
    Str s;
    s.w = w;
    uint32_t p = 0;
    for (uint32_t i = 0; i < w.size(); ++i) {
        s.st.push_back(p);
        const uint32_t c = wgroups(w[i]);
        s.cov.insert(s.cov.end(), c, i);
        p += c;
    }
    return s;
}
bool zero_fill(uint32_t w) { return is_fill(w) && !fill_bit(w); }
bool one_fill(uint32_t w) { return is_fill(w) && fill_bit(w); }
// a literal of y covering one of the groups [a, b)
bool literal_in(const Str& Y, uint32_t a, uint32_t b) {
    for (uint32_t g = a; g < b; ++g)
        if (!is_fill(Y.w[Y.cov[g]])) return true;
    return false;
}
// "-": x's 0-fill i, begun before y's word at group q, is counted over q
bool counted(const Str& X, const Str& Y, int i, uint32_t q) {
    while (true) {
        const uint32_t a = X.st[i];
        const int j = (int)Y.cov[q] - 1;
        if (j < 0) return true;
        const uint32_t c = Y.st[j];
        if (!(one_fill(Y.w[j]) && c < a)) return true;
        if (i == 0 || !(zero_fill(X.w[i - 1]) && X.st[i - 1] < c)) return false;
        --i;
        q = c;
    }
}
bool flag(int op, const Str& X, const Str& Y, uint32_t p, uint32_t G) {
    const uint32_t i = X.cov[p], j = Y.cov[p];
    const bool xe = p + 1 == G || X.st[X.cov[p + 1]] == p + 1, ye = p + 1 == G || Y.st[Y.cov[p + 1]] == p + 1;
    const uint32_t absorb = op == OP_OR ? 1u : 0u;
    switch (single_flag(op, X.w[i], Y.w[j], X.st[i] == p, Y.st[j] == p, xe, ye)) {
    case SF_NO: return false;
    case SF_YES: return true;
    case SF_WALK_AND_X:
        return !(i > 0 && is_fill(X.w[i - 1]) && fill_bit(X.w[i - 1]) == absorb && X.st[i - 1] < Y.st[j] &&
                 literal_in(Y, X.st[i - 1], Y.st[j]));
    case SF_WALK_AND_Y: return literal_in(Y, X.st[i], p);
    case SF_WALK_MINUS_X:
        return !(i > 0 && zero_fill(X.w[i - 1]) && X.st[i - 1] < Y.st[j] && counted(X, Y, (int)i - 1, Y.st[j]));
    default: {
        if (j == 0 || !one_fill(Y.w[j - 1]) || Y.st[j - 1] >= X.st[i]) return true;
        const uint32_t c = Y.st[j - 1];
        return i > 0 && zero_fill(X.w[i - 1]) && X.st[i - 1] < c && counted(X, Y, (int)i - 1, c);
    }
    }
}
void by_groups(int op, const V& xw, const V& yw, uint32_t G, V& out) {
    const Str X = expand(xw), Y = expand(yw);
    std::vector<uint32_t> r(G);
    for (uint32_t g = 0; g < G; ++g) r[g] = apply_op(op, wpattern(xw[X.cov[g]]), wpattern(yw[Y.cov[g]]));
    for (uint32_t g = 0; g < G;) {
        const uint32_t c = cls_of(r[g]);
        uint32_t e = g + 1;
        if (c != C_MIXED) while (e < G && r[e] == r[g]) ++e;
        out.push_back(run_word(c, e - g, r[g], c != C_MIXED && e == g + 1 && flag(op, X, Y, g, G)));
        g = e;
    }
}
}  // namespace

// Pairs of random operands (fills of any length and value, neighbours equal
// or not, count-1 fills, lone uniform literals) whose words differ, for `op`.
extern "C" long group_model_mismatches(int op, unsigned seed, long pairs) {
    std::mt19937 rng(seed);
    auto R = [&](uint32_t n) { return (uint32_t)(rng() % n); };
    long bad = 0;
    for (long it = 0; it < pairs; ++it) {
        const uint32_t G = 2 + R(it % 3 == 0 ? 8 : it % 3 == 1 ? 40 : 300);
        V w[2];
        for (V& v : w) {
            const uint32_t pf = R(100), p1 = R(100), maxc = 2 + R(12), pl = R(101);
            for (uint32_t g = 0; g < G;) {
                if (R(100) < pf) {
                    const uint32_t c = std::min(G - g, R(100) < p1 ? 1u : 1 + R(maxc));
                    v.push_back((R(2) ? HEADER1 : HEADER0) | c);
                    g += c;
                } else {
                    v.push_back(R(100) < pl ? 1 + R(0x7ffffffe) : R(2) ? 0u : ALLONES);
                    ++g;
                }
            }
        }
        V a, b;
        merge(op, true, w[0], w[1], G, a, (unsigned)it);
        by_groups(op, w[0], w[1], G, b);
        bad += a != b;
    }
    return bad;
}
