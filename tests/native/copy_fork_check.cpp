// mk::copy_out in a child that was forked while other threads wake the helpers
// and copy: the child has no helpers and whatever locks were held stay held in
// its memory.  Every child ends, with its bytes.
#include <stdio.h>
#include <string.h>
#include <sys/wait.h>
#include <unistd.h>

#include <atomic>
#include <thread>
#include <vector>

#include "mk_internal.h"

constexpr size_t kBytes = 400000;

static bool copies(int n) {
    std::vector<unsigned char> src(kBytes), dst(kBytes);
    for (size_t i = 0; i < kBytes; ++i) src[i] = (unsigned char)((i * 2654435761u) >> 13);
    for (int i = 0; i < n; ++i) {
        memset(dst.data(), 0, kBytes);
        mk::copy_out_soon(kBytes);
        mk::copy_out(dst.data(), src.data(), kBytes);
        if (memcmp(dst.data(), src.data(), kBytes) != 0) return false;
    }
    return true;
}

int main() {
    if (!copies(3)) return printf("before the fork\n"), 1;
    std::atomic<bool> stop{false};
    std::vector<std::thread> ts;
    for (int t = 0; t < 6; ++t)
        ts.emplace_back([&stop] {
            while (!stop) {
                for (int i = 0; i < 100; ++i) mk::copy_out_soon(kBytes);
                copies(1);
            }
        });
    int bad = 0;
    for (int i = 0; i < 150 && !bad; ++i) {
        const pid_t pid = fork();
        if (pid == 0) {
            alarm(5);
            _exit(copies(4) ? 0 : 1);
        }
        int st = 0;
        waitpid(pid, &st, 0);
        if (!WIFEXITED(st) || WEXITSTATUS(st) != 0) bad = i + 1;
    }
    stop = true;
    for (auto &t : ts) t.join();
    if (bad) return printf("child %d\n", bad), 1;
    if (!copies(3)) return printf("after the forks\n"), 1;
    printf("ok\n");
    return 0;
}
