// mk::div_by against the division, bit for bit, over quotients, divisors with
// extreme significands and the sizes planes and CPR rows divide by.
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "mk_math.h"

static uint64_t s = 88172645463325252ull;
static uint64_t rnd() {
    s ^= s << 13;
    s ^= s >> 7;
    return s ^= s << 17;
}

int main() {
    for (long i = 0; i < 20000000; ++i) {
        uint32_t ua = ((uint32_t)rnd() & 0x807fffffu) | (uint32_t)(107 + rnd() % 40) << 23;
        uint32_t ud = ((uint32_t)rnd() & 0x007fffffu) | (uint32_t)(117 + rnd() % 20) << 23;
        if (i % 7 == 0) ud |= 0x7fffffu;
        if (i % 11 == 0) ud &= 0xff800001u;
        if (i % 13 == 0) ua |= 0x7ffffeu;
        float a, d;
        memcpy(&a, &ua, 4);
        memcpy(&d, &ud, 4);
        if (mk::div_by(a, d, 1.0f / d) != a / d) return printf("float %a / %a\n", a, d), 1;
    }
    for (long i = 0; i < 10000000; ++i) {
        const uint64_t ua = (rnd() & 0x800fffffffffffffull) | (uint64_t)(1003 + rnd() % 40) << 52;
        double a;
        memcpy(&a, &ua, 8);
        const double d = (double)(1 + (i < 5000000 ? i % 16384 : (long)(rnd() % 2147483647u)));
        if (mk::div_by(a, d, 1.0 / d) != a / d) return printf("double %a / %a\n", a, d), 1;
    }
    printf("ok\n");
    return 0;
}
