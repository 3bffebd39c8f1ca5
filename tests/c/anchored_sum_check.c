/* Host check of the float-pair anchored sum (the algorithm of df32.cuh's
 * anchor_add / dfa_first / dfa_add / dfa_end / dfa_renorm, restated in C with
 * the C library's correctly rounded fmaf).  On random stencil sums of float
 * pairs it verifies
 *   - every step q = T_k - T_{k-1} and the closing T_n - sigma are exact,
 *   - the closing Fast2Sum is exact,
 *   - the final pair is within n^2 2^-46 B of the exact sum (binary128),
 *     B = sum |ch_k| |xh_k|, the bound the library states.
 * Prints the largest error / B per term count and exits non-zero on a
 * violation.
 *
 * Usage: anchored_sum_check <trials> <seed>
 * Build: gcc -O2 -ffp-contract=off anchored_sum_check.c -lm
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#if defined(__aarch64__)
typedef long double quad; /* binary128 */
#else
typedef __float128 quad;
#endif

static uint64_t rng_state;
static uint64_t next_u64(void) { /* SplitMix64 */
    uint64_t z = (rng_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double uniform(void) { return (double)(next_u64() >> 11) * (1.0 / 9007199254740992.0); }

static void split(double x, float *h, float *l) {
    *h = (float)x;
    *l = (float)(x - (double)*h);
}

int main(int argc, char **argv) {
    const long trials = argc > 1 ? atol(argv[1]) : 200000;
    rng_state = argc > 2 ? strtoull(argv[2], 0, 10) : 1;
    const int sizes[] = {3, 5, 7, 9, 13, 19};
    double worst[6] = {0};
    long bad = 0;
    for (long t = 0; t < trials; ++t) {
        const int si = (int)(t % 6), n = sizes[si];
        float ch[19], cl[19], xh[19], xl[19];
        /* mixed or single signs, magnitudes spread over up to 2^79; every
           fifth case one dominant term of the sign opposite to the rest */
        const int mixed_c = (t / 6) % 2, mixed_x = (t / 12) % 2, spread = (int)((t / 24) % 4) * 13;
        const int big = t % 5 == 0 ? (int)(next_u64() % (uint64_t)n) : -1;
        for (int k = 0; k < n; ++k) {
            double c = ldexp(0.5 + uniform(), -(int)(uniform() * 8));
            if (mixed_c && uniform() < 0.5) c = -c;
            double x = ldexp(0.5 + uniform(), -(int)(uniform() * spread)) * ldexp(1.0, (int)(uniform() * 40) - 20);
            if (mixed_x && uniform() < 0.5) x = -x;
            if (k == big) x *= -ldexp(1.0, (int)(uniform() * 30));
            split(c, &ch[k], &cl[k]);
            split(x, &xh[k], &xl[k]);
        }
        float b = 0.0f, sg = 0.0f;
        for (int k = 0; k < n; ++k) {
            b = fmaf(fabsf(ch[k]), fabsf(xh[k]), b);
            sg = fmaf(2.0f * (1.0f + 0x1p-15f) * fabsf(ch[k]), fabsf(xh[k]), sg);
        }
        float tk = sg, hi = 0.0f, lo = 0.0f;
        for (int k = 0; k < n; ++k) {
            const float tn = fmaf(ch[k], xh[k], tk);
            const float q = tn - tk;
            if ((double)q != (double)tn - (double)tk) {
                if (bad++ < 5) fprintf(stderr, "trial %ld term %d: T_k - T_(k-1) not exact\n", t, k);
            }
            const float r = fmaf(ch[k], xh[k], -q);
            hi = k == 0 ? r : hi + r;
            lo = k == 0 ? fmaf(cl[k], xh[k], ch[k] * xl[k]) : fmaf(cl[k], xh[k], fmaf(ch[k], xl[k], lo));
            tk = tn;
        }
        const float h = tk - sg, l = hi + lo;
        if ((double)h != (double)tk - (double)sg) {
            if (bad++ < 5) fprintf(stderr, "trial %ld: T_n - sigma not exact\n", t);
        }
        const float s = h + l, e = l - (s - h);
        if ((quad)s + (quad)e != (quad)h + (quad)l) {
            if (bad++ < 5) fprintf(stderr, "trial %ld: closing Fast2Sum not exact (h %a l %a)\n", t, h, l);
        }
        quad ex = 0;
        for (int k = 0; k < n; ++k) ex += ((quad)ch[k] + (quad)cl[k]) * ((quad)xh[k] + (quad)xl[k]);
        quad err = (quad)s + (quad)e - ex;
        if (err < 0) err = -err;
        const double rel = b > 0 ? (double)(err / (quad)b) : 0.0;
        if (rel > worst[si]) worst[si] = rel;
        if (rel > (double)n * n * 0x1p-46) {
            if (bad++ < 5) fprintf(stderr, "trial %ld (n=%d): error %.3e B\n", t, n, rel);
        }
    }
    for (int i = 0; i < 6; ++i) printf("n=%d worst_error_over_B=%.3e bound=%.3e\n", sizes[i], worst[i],
                                       (double)sizes[i] * sizes[i] * 0x1p-46);
    printf("violations=%ld\n", bad);
    return bad ? 1 : 0;
}
