/*
 * b2g_lists.h — places of lists that share one array, counted in 64 bits: what a query finds in all may be
 * past 31 bits, and lists that do not fit must be seen not to, whatever the total.
 */
#ifndef B2G_LISTS_H
#define B2G_LISTS_H

#include <limits.h>
#include <stdint.h>

#include "b2g_trig.h" /* B2G_HD */

namespace b2g {

/* whether `count` entries from `first` on lie in an array of `cap` */
B2G_HD bool list_fits(unsigned long long first, int count, int cap) {
    return count >= 0 && cap >= 0 && first <= (unsigned long long)cap && (unsigned long long)count <= (unsigned long long)cap - first;
}

/* a total as the 32-bit count of an entry point: one past them all reads as the largest */
B2G_HD int32_t saturated_count(unsigned long long total) { return total > (unsigned long long)INT32_MAX ? INT32_MAX : (int32_t)total; }

/* whether a total fits a caller's capacity */
B2G_HD bool within_capacity(unsigned long long total, int32_t capacity) { return capacity >= 0 && total <= (unsigned long long)capacity; }

}  // namespace b2g

#endif
