// mk::add_steps against a loop of float additions.  Prints "ok <cases>" or the
// first difference.
#include <initializer_list>
#include <stdio.h>

#include "mk_math.h"

int main() {
    long n_cases = 0;
    for (int dim = 1; dim <= 5000; dim += dim < 300 ? 1 : 37) {
        const float one = 1.0f / (float)dim;
        for (float step : {one, one / 4, one / 8}) {
            for (int k = 0; k < 60; ++k) {
                // anywhere on the schedule's range, below it, and next to powers of two
                float a = (float)((k * 7919 % 1000) / 1000.0 * 1.8) - 0.02f;
                if (k % 3 == 0)
                    for (int i = 0; i < k; ++i) a += step;
                if (k % 5 == 0) a = (k % 2 ? 0.25f : 1.0f) - (float)(k / 2) * step;
                for (int n : {0, 1, 2, 3, 4, 5, 6, 7, 15, 31, 63, 100, 241}) {
                    float want = a;
                    for (int i = 0; i < n; ++i) want += step;
                    const float got = mk::add_steps(a, step, n);
                    if (got != want) {
                        printf("a %a step %a n %d: %a, want %a\n", a, step, n, got, want);
                        return 1;
                    }
                    ++n_cases;
                }
            }
        }
    }
    // steps that fall halfway between two floats of the range
    for (int e = -6; e <= 0; ++e) {
        const float ulp = ldexpf(1.0f, e - 23);
        for (int q = 0; q < 64; ++q) {
            const float step = ((float)q + 0.5f) * ulp;
            for (int k = 0; k < 64; ++k) {
                const float a = ldexpf(1.0f, e) + (float)k * ulp;
                for (int n : {5, 6, 9, 30, 240}) {
                    float want = a;
                    for (int i = 0; i < n; ++i) want += step;
                    if (mk::add_steps(a, step, n) != want) {
                        printf("halfway: a %a step %a n %d\n", a, step, n);
                        return 1;
                    }
                    ++n_cases;
                }
            }
        }
    }
    printf("ok %ld\n", n_cases);
    return 0;
}
