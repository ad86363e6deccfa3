// Raw column values as unsigned keys in value order, so that a range term's
// comparison of a row (qContinuousRange::inRange in double, src/qExpr.cpp:
// 1647-1667) is one subtraction and one unsigned comparison on the device.
// The bounds in keys are found on the host by searching the keys with the
// double comparison itself, so both agree on every value, NaN (never inside a
// bounded range) and the two zeros included.
#ifndef WAH_KEYS_H
#define WAH_KEYS_H
#include <stdint.h>
#include <string.h>
#include "wah_core.cuh"

namespace wah {

// key = v ^ ((v >> 31, arithmetic) & flip | sign): 0 uint32, 1 float32, 2 int32
struct KeyMap { uint32_t flip, sign; };
WAH_HD KeyMap key_map(uint32_t vtype) {
    KeyMap m;
    m.flip = vtype == 1u ? 0xFFFFFFFFu : 0u;
    m.sign = vtype == 0u ? 0u : 0x80000000u;
    return m;
}
WAH_HD uint32_t value_key(uint32_t v, KeyMap m) {
    return v ^ (((uint32_t)((int32_t)v >> 31) & m.flip) | m.sign);
}

inline double key_value(uint32_t key, uint32_t vtype) {
    if (vtype == 0u) return (double)key;
    if (vtype == 2u) return (double)(int32_t)(key ^ 0x80000000u);
    const uint32_t b = key & 0x80000000u ? key ^ 0x80000000u : ~key;
    float f;
    memcpy(&f, &b, 4);
    return (double)f;
}
// Keys [lo, lo + span] of the values with `vlo lop x rop vhi` (0 none, 1 <,
// 2 <=); false when no value is inside.
inline bool key_range(uint32_t vtype, uint32_t lop, double vlo, uint32_t rop, double vhi, uint32_t& lo, uint32_t& span) {
    // -inf .. +inf; NaN keys lie outside
    const uint64_t kmin = vtype == 1u ? 0x007FFFFFull : 0ull, kmax = vtype == 1u ? 0xFF800000ull : 0xFFFFFFFFull;
    uint64_t a = kmin, b = kmax + 1;  // first key passing the lower side
    while (a < b) {
        const uint64_t m = (a + b) / 2;
        const double v = key_value((uint32_t)m, vtype);
        if (lop == 0 || (lop == 1 ? vlo < v : vlo <= v)) b = m; else a = m + 1;
    }
    uint64_t c = kmin, d = kmax + 1;  // first key failing the upper side
    while (c < d) {
        const uint64_t m = (c + d) / 2;
        const double v = key_value((uint32_t)m, vtype);
        if (rop == 0 || (rop == 1 ? v < vhi : v <= vhi)) c = m + 1; else d = m;
    }
    if (a >= c) return false;
    lo = (uint32_t)a;
    span = (uint32_t)(c - 1 - a);
    return true;
}

}  // namespace wah
#endif
