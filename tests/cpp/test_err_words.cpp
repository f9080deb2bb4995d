// err_words.h: a word a holder, errors stay with the one they belong to, holders beyond the last word share word 0
#include <cstdio>
#include <vector>

#include "../../turboinfer_b200/csrc/err_words.h"

static int g_fail = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++g_fail; } } while (0)

int main() {
    static tib::ErrWords w;
    CHECK(!w.fetch(0));   // (no memory yet)
    std::vector<int> mem(tib::ErrWords::kWords, 0);
    w.host = mem.data();
    const int a = w.take(), b = w.take();
    CHECK(a > 0 && b > 0 && a != b);
    mem[b] = 1;           // b's kernels gave up
    CHECK(!w.fetch(0) && !w.fetch(a));
    CHECK(w.fetch(b) && !w.fetch(b));
    mem[a] = 1;           // ... and a's, whose holder goes without looking
    w.give(a);
    CHECK(w.take() == a && !w.fetch(a));
    int n = 2;
    while (w.take() > 0) ++n;
    CHECK(n == tib::ErrWords::kWords - 1);
    w.give(b);
    CHECK(w.take() == b && w.take() == 0);
    return g_fail ? 1 : 0;
}
