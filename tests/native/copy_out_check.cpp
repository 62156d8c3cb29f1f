// mk::copy_out from several threads at once, with and without a wake, and in
// a forked child (which has no helpers): every byte arrives, none beside them.
#include <stdio.h>
#include <string.h>
#include <sys/wait.h>
#include <unistd.h>

#include <thread>
#include <vector>

#include "mk_internal.h"

static bool round_trip(size_t n, unsigned seed, bool wake) {
    std::vector<unsigned char> src(n), dst(n + 2, 0xEE);
    for (size_t i = 0; i < n; ++i) src[i] = (unsigned char)((i * 2654435761u + seed) >> 13);
    if (wake) mk::copy_out_soon(n);
    mk::copy_out(dst.data() + 1, src.data(), n);
    return dst[0] == 0xEE && dst[n + 1] == 0xEE && (n == 0 || memcmp(dst.data() + 1, src.data(), n) == 0);
}

static bool many(unsigned seed) {
    bool ok = true;
    for (int r = 0; r < 6; ++r)
        for (size_t n : {(size_t)0, (size_t)1, (size_t)262143, (size_t)262144, (size_t)262145, (size_t)524288,
                         (size_t)1000003, (size_t)3145728})
            ok = ok && round_trip(n, seed + r, (r & 1) != 0);
    return ok;
}

// Copies close together, each larger than the one before: helpers are late for
// one and meet the next.
static bool close_together() {
    std::vector<unsigned char> src(786432), dst(786432);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (unsigned char)((i * 2654435761u) >> 13);
    for (int r = 0; r < 20000; ++r) {
        const size_t n = 262144 + (size_t)(r % 9) * 65536;
        dst[n - 1] = (unsigned char)~src[n - 1];
        mk::copy_out_soon(n);
        mk::copy_out(dst.data(), src.data(), n);
        if (dst[n - 1] != src[n - 1] || dst[0] != src[0]) return false;
        dst[0] = (unsigned char)~src[0];
    }
    return memcmp(dst.data() + 1, src.data() + 1, dst.size() - 1) == 0;
}

int main() {
    if (!close_together()) return printf("close together\n"), 1;
    if (!many(1)) return printf("one thread\n"), 1;
    bool ok[6];
    std::vector<std::thread> ts;
    for (int t = 0; t < 6; ++t) ts.emplace_back([&ok, t] { ok[t] = many(100u * t); });
    for (auto &t : ts) t.join();
    for (bool b : ok)
        if (!b) return printf("several threads\n"), 1;
    fflush(stdout);
    const pid_t pid = fork();
    if (pid == 0) _exit(many(7) ? 0 : 1);
    int st = 0;
    waitpid(pid, &st, 0);
    if (!WIFEXITED(st) || WEXITSTATUS(st) != 0) return printf("after fork\n"), 1;
    printf("ok\n");
    return 0;
}
