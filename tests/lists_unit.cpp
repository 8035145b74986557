/* lists_unit.cpp — the places of a query's lists (b2g_lists.h) at totals around 2^31 and 2^32. */
#include <cstdio>
#include <initializer_list>

#include "b2g_lists.h"

using namespace b2g;

static int failures = 0;
static void check(bool ok, const char* what) {
    if (!ok) {
        std::printf("wrong: %s\n", what);
        ++failures;
    }
}

int main() {
    const unsigned long long k31 = 1ull << 31, k32 = 1ull << 32;
    check(list_fits(0, 0, 0) && list_fits(0, 16, 16) && list_fits(15, 1, 16) && list_fits(16, 0, 16), "lists that fit");
    check(!list_fits(0, 17, 16) && !list_fits(16, 1, 16) && !list_fits(17, 0, 16), "lists one too long");
    check(list_fits(INT_MAX - 4, 4, INT_MAX) && !list_fits(INT_MAX - 3, 4, INT_MAX), "lists at the largest room");
    /* places that are negative, or small again, in 32 bits */
    for (unsigned long long base : {k31, k31 + 1, k32 - 1, k32, k32 + 7, 5 * k32 + 100})
        check(!list_fits(base, 1, 1 << 24) && !list_fits(base, 250000, INT_MAX), "places past the room");
    /* the adds of 8600 boxes over 250,000 fixtures: only those within the room are written */
    const int count = 250000, cap = 16 * 8600;
    unsigned long long total = 0;
    long long written = 0;
    for (int i = 0; i < 20000; ++i) {
        if (list_fits(total, count, 8 * count)) written += count;
        check(!list_fits(total, count, cap), "no room for the first list already");
        total += (unsigned long long)count;
    }
    check(written == 8ll * count, "eight lists of room for eight");
    check(total > k32, "the total passes 32 bits");
    check(saturated_count(total) == INT32_MAX && saturated_count(k31) == INT32_MAX && saturated_count(k31 - 1) == INT32_MAX, "saturated");
    check(saturated_count(0) == 0 && saturated_count(12345) == 12345, "small totals as they are");
    for (unsigned long long t : {k31, k32 - 5, k32, k32 + 3, total})
        check(!within_capacity(t, INT_MAX) && !within_capacity(t, 64), "totals past every capacity");
    check(within_capacity(0, 0) && within_capacity(64, 64) && !within_capacity(65, 64) && !within_capacity(0, -1), "capacities");
    std::printf("%d wrong\n", failures);
    return failures != 0;
}
