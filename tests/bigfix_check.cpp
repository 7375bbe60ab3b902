// bigfix_check.cpp -- bigfix_mul (csrc/bigfix.h) against the schoolbook product
// with every limb product, on random and extreme limbs.  Prints the number of
// products that differ.
#include <cstdio>
#include <random>

#include "../chaos-ultra_gb300/csrc/bigfix.h"

int main()
{
    std::mt19937_64 r(5);
    long bad = 0;
    for (int it = 0; it < 200000; it++) {
        const int L = 1 + (int)(r() % chaos::BIGFIX_MAX_LIMBS);
        chaos::BigFix a = chaos::bigfix_zero(L), b = chaos::bigfix_zero(L);
        for (int k = 0; k <= L; k++) {
            const unsigned m = r() % 4, n = r() % 4;  // all ones, zero or random
            a.w[k] = m == 0 ? ~0ull : m == 1 ? 0 : r();
            b.w[k] = n == 0 ? ~0ull : n == 1 ? 0 : r();
        }
        a.w[L] &= 3, b.w[L] &= 3;
        a.neg = r() & 1, b.neg = r() & 1;
        uint64_t p[2 * chaos::BIGFIX_MAX_LIMBS + 3] = {};
        for (int i = 0; i <= L; i++) {
            unsigned __int128 carry = 0;
            for (int j = 0; j <= L; j++) {
                const unsigned __int128 t = (unsigned __int128)a.w[i] * b.w[j] + p[i + j] + carry;
                p[i + j] = (uint64_t)t;
                carry = t >> 64;
            }
            p[i + L + 1] = (uint64_t)carry;
        }
        const chaos::BigFix q = chaos::bigfix_mul(a, b);
        bool same = q.neg == (a.neg != b.neg && !q.is_zero());
        for (int k = 0; k <= L; k++) same = same && q.w[k] == p[k + L];
        bad += !same;
    }
    std::printf("%ld\n", bad);
    return 0;
}
