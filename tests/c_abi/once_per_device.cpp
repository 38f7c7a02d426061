// OncePerDevice: pending on every device until set on that one.
#include <cstdio>

#include "xmc_internal.h"

int main() {
    xmc::OncePerDevice once;
    for (int d : {0, 1, 7, 63, 64, 200})
        if (!once.pending(d)) return 1;
    once.set(0);
    if (once.pending(0) || !once.pending(1) || !once.pending(63)) return 2;
    once.set(63);
    once.set(1);
    if (once.pending(63) || once.pending(1) || !once.pending(2) || !once.pending(62)) return 3;
    once.set(64);
    if (!once.pending(64) || once.pending(0) || !once.pending(2)) return 4;
    xmc::OncePerDevice other;
    if (!other.pending(0)) return 5;
    std::puts("ok");
    return 0;
}
