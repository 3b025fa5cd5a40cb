/* Launch shape of mixed-radix lines (kernels/fft_mr.cuh): radix list, digit
 * strides with their bank padding, transforms and threads per CTA (C99). */
#include <math.h>
#include <string.h>

#include "fz_internal.h"

/* Issue slots of one radix-R butterfly: the codelet's arithmetic, about ten a
 * value for its shared-memory accesses, twiddle and addresses, and the index
 * maps. 0: no butterfly of that radix. */
static int mr_cost(int R)
{
    static const int flops[17] = {0, 0, 4, 16, 16, 44, 44, 100, 56, 112, 108, 240, 112, 330, 228, 212, 168};
    return R >= 1 && R <= 16 ? flops[R] + 10 * R + 12 : 0;
}

typedef struct
{
    int min_stages, pair;
    int cur[FFTZ_MR_STAGES], best[FFTZ_MR_STAGES];
    int nbest;
    double score;
} mr_search;

static void mr_try(mr_search *q, int64_t rest, int depth, int top, double cost)
{
    if (rest == 1)
    {
        if (q->pair && depth > 1 && q->cur[depth - 1] > 8) return;
        if (depth >= q->min_stages && (q->nbest == 0 || cost < q->score))
        {
            q->score = cost;
            q->nbest = depth;
            memcpy(q->best, q->cur, sizeof(int) * (size_t)depth);
        }
        return;
    }
    if (depth == FFTZ_MR_STAGES || (q->nbest && cost >= q->score)) return;
    for (int R = top; R >= 2; R--)
        if (rest % R == 0)
        {
            q->cur[depth] = R;
            /* three slots a value stand for the stage's barrier */
            mr_try(q, rest / R, depth + 1, R, cost + (double)mr_cost(R) / R + 3.0);
        }
}

/* Radices (largest first) of the cheapest split of n into at least min_stages
 * stages, the last of at most 8 for pair (real lines, whose last stage holds two
 * butterflies a thread); returns their number, 0 when n has a prime factor above
 * 13. cost (may be NULL): issue slots a point. */
int fz_mr_radices(int64_t n, int min_stages, int pair, int32_t *radix, double *cost)
{
    mr_search q;
    memset(&q, 0, sizeof(q));
    q.min_stages = min_stages;
    q.pair = pair;
    int64_t m = n;
    static const int pr[] = {2, 3, 5, 7, 11, 13};
    for (int i = 0; i < 6; i++)
        while (m % pr[i] == 0) m /= pr[i];
    if (n == 1)
    {
        radix[0] = 1; /* a copy */
        if (cost) *cost = 0;
        return 1;
    }
    if (n < 2 || m != 1) return 0;
    mr_try(&q, n, 0, 16, 0.0);
    if (!q.nbest && pair) /* nothing but 11 and 13 */
    {
        q.pair = 0;
        mr_try(&q, n, 0, 16, 0.0);
    }
    for (int s = 0; s < q.nbest; s++) radix[s] = q.best[s];
    if (cost) *cost = q.score;
    return q.nbest;
}

static uint32_t magic(int64_t d) { return d <= 1 ? 0u : (uint32_t)((0xFFFFFFFFull + (uint64_t)d) / (uint64_t)d); }

/* slots of one line with `pad` extra per digit-0 block */
static int64_t mr_span(const fftz_pass_t *k, int pad) { return k->n + (int64_t)pad * (k->nstages > 1 ? k->radix[0] : 0); }

/* Most lines of this length a CTA can hold (0: none). */
static int64_t mr_lines(const fftz_pass_t *k, int64_t cap)
{
    const int64_t esz = k->dtype == 0 ? 8 : 16;
    const int64_t per = (k->sstride + ((k->flags & FFTZ_F_TW4) ? 16 : 0)) * esz + 32;
    return cap / per;
}

/* 1 if a line of n points fits cap bytes of shared memory as a mixed-radix tile
 * (a product of the primes up to 13 that fits never needs more stages than there
 * are: 5^6 takes six). */
int fz_mr_fits(int dtype, int64_t n, int64_t cap)
{
    const int64_t esz = dtype == 0 ? 8 : 16;
    if (n < 1 || (n + 1 + 16) * esz + 32 > cap) return 0;
    static const int pr[] = {2, 3, 5, 7, 11, 13};
    for (int i = 0; i < 6; i++)
        while (n % pr[i] == 0) n /= pr[i];
    return n == 1;
}

/* the smallest product of 2, 3, 5 and 7 that is at least n */
static int64_t next_smooth7(int64_t n)
{
    for (;; n++)
    {
        int64_t m = n;
        while (m % 2 == 0) m /= 2;
        while (m % 3 == 0) m /= 3;
        while (m % 5 == 0) m /= 5;
        while (m % 7 == 0) m /= 7;
        if (m == 1) return n;
    }
}

/* Rounding error of a chirp-z transform of n points over a convolution of m
 * points: rel-L2^2 = 48 + (2 n / m) X, in 1e-16 (float; double in 2^-58 of that). The
 * noise of both FFTs is white over the m points and the n wanted ones hold half
 * of the signal, hence 2 n / m: padding lowers the error. X is the sum below over the
 * stages of both FFTs, fitted on B200 to 1426 pairs of n (17 ... 400009) and m in float
 * (residual 1.7% of rel-L2^2); double has the same, plus the error of a spectrum
 * formed in double where it is (tables.c). */
static double blue_noise(int nst, const int32_t *radix, int64_t m)
{
    static const double butterfly[17] = {0, 0, 0, 0.3, 0, 7.4, 4.7, 12.1, 8.0, 18.4, 13.3, 0, 11.0, 0, 17.6, 21.0, 17.1};
    double x = 0;
    for (int s = 0; s < nst; s++)
    {
        m /= radix[s];
        x += 2 * butterfly[radix[s]];
        if (s < nst - 1) x += 2 * 36.1 * (1 - 1.0 / radix[s]) * (1 - 1.0 / (double)m);
    }
    return x;
}

/* 1 if a convolution of m points with stage noise x is no less exact (to 1%) than
 * one over the power of two, as it ran before lengths with odd factors were taken:
 * X per bit measured by the bit length of that power of two (above 2^14 float and
 * 2^13 double in three passes). A power of two itself always is. */
static int blue_exact_enough(int dtype, int64_t n, int64_t m, double x)
{
    static const double former[2][21] = {
        {0, 0, 0, 0, 0, 0, 19.5, 19.5, 23.2, 22.7, 23.2, 24.9, 27.0, 24.9, 26.2, 31.2, 31.2, 31.2, 31.2, 31.2, 31.2},
        {0, 0, 0, 0, 0, 0, 21.0, 29.0, 33.0, 40.0, 40.5, 41.0, 41.0, 48.0, 48.6, 49.4, 47.9, 51.0, 54.0, 56.0, 54.0}};
    int l = 6;
    while (((int64_t)1 << l) < 2 * n - 1) l++;
    const double p = (double)((int64_t)1 << l);
    if ((double)m >= p) return 1;
    /* the former kernels' gain error (fz_mr_gain) is not divided by the padding */
    double limit = former[dtype == 0 ? 0 : 1][l < 20 ? l : 20] * l * (2.0 * (double)n < 0.56 * p ? 1.1 : 1.0);
    if (dtype == 1) x += m <= FZ_EXACT_SPECTRUM ? 10 : 19.5 * log2((double)m);
    return (22.6 + x) * p <= 1.03 * limit * (double)m;
}

/* Convolution length of a chirp-z transform of n points in one tile: of the
 * 7-smooth m >= 2n - 1 that are exact enough, from the first on up to a quarter
 * beyond it, the one with the fewest issue slots over both sweeps (a longer m with
 * fewer stages beats the nearest one); 0 when none fits cap bytes. */
int64_t fz_mr_blue_len(int dtype, int64_t n, int64_t cap)
{
    int32_t r[FFTZ_MR_STAGES];
    int64_t best = 0, last = INT64_MAX;
    double score = 0, c;
    const int64_t need = 2 * n - 1;
    for (int64_t m = next_smooth7(need < 4 ? 4 : need); m <= last && fz_mr_fits(dtype, m, cap); m = next_smooth7(m + 1))
    {
        const int nst = fz_mr_radices(m, 2, 0, r, &c);
        if (nst < 2 || (best && (double)m * c >= score) || !blue_exact_enough(dtype, n, m, blue_noise(nst, r, m))) continue;
        if (!best) last = m + m / 4 + 4;
        best = m;
        score = (double)m * c;
    }
    return best;
}

/* Convolution length m = n1 * n2 of a chirp-z transform in three passes: the
 * cheapest of the first twelve 7-smooth lengths from 2n - 1 on that are exact enough
 * and have both factors one tile, n2 of at least two stages, within a factor of
 * four of each other (any such length when none is exact enough). */
int64_t fz_mr_blue_split(int dtype, int64_t n, int64_t cap, int64_t *n1, int64_t *n2)
{
    int32_t ra[FFTZ_MR_STAGES], rb[FFTZ_MR_STAGES];
    int64_t best = 0;
    double score = 0, ca, cb;
    for (int strict = 1; strict >= 0 && !best; strict--)
    {
        int64_t m = 2 * n - 2;
        for (int found = 0, tries = 0; found < 12 && tries < (strict ? 1000 : 64); tries++)
        {
            m = next_smooth7(m + 1);
            if (strict && m > 4 * n) break;
            int any = 0;
            for (int64_t a = 2; a * a <= 4 * m; a++)
            {
                const int64_t b = m / a;
                if (m % a || a > 4 * b || b > 4 * a || !fz_mr_fits(dtype, a, cap) || !fz_mr_fits(dtype, b, cap)) continue;
                const int sa = fz_mr_radices(a, 1, 0, ra, &ca), sb = fz_mr_radices(b, 2, 0, rb, &cb);
                if (sa < 1 || sb < 2) continue;
                /* 90: the four-step factors between the passes */
                if (strict && !blue_exact_enough(dtype, n, m, 90 + blue_noise(sa, ra, a) + blue_noise(sb, rb, b))) continue;
                any = 1;
                if (!best || (double)m * (ca + cb) < score)
                {
                    best = m;
                    score = (double)m * (ca + cb);
                    *n1 = a;
                    *n2 = b;
                }
            }
            found += any;
        }
    }
    return best;
}

/* Slot of item i (of one line, or of tpc lines when col) of stage s; first /
 * last are the maps of the HBM-side stages. */
static int mr_addr(const fftz_pass_t *k, int s, int i, int col)
{
    const int S = k->nstages;
    const int R = k->radix[s], M = k->mr.st[s].m, nb = k->n / R;
    int p, x;
    if (col)
    {
        x = i / k->tpc;
        p = i % k->tpc;
    }
    else
    {
        p = i / nb;
        x = i % nb;
    }
    const int base = p * k->sstride;
    if (s == 0) return base + x;
    if (s == S - 1)
    {
        int o = 0;
        for (int j = 0; j < S - 1; j++)
        {
            o += (x % k->radix[j]) * (k->mr.st[j].m + (j == 0 ? k->mr.pad : 0));
            x /= k->radix[j];
        }
        return base + o;
    }
    const int b = x / M;
    int B = 1;
    for (int j = 1; j < s; j++) B *= k->radix[j];
    return base + x + b * M * (R - 1) + (b / B) * k->mr.pad;
}

/* Shared-memory wavefronts per lane group (16 float or 8 double slots span all
 * banks) over the first groups of every stage, for the pad and stride in k; stops
 * counting at most. */
static int mr_conflicts(const fftz_pass_t *k, int most)
{
    const int W = k->dtype == 0 ? 16 : 8;
    int tot = 0;
    for (int s = 0; s < k->nstages; s++)
    {
        const int col = (s == 0 && k->in_mode == 1) || (s == k->nstages - 1 && k->out_mode == 1);
        const int items = k->tpc * (k->n / k->radix[s]);
        for (int g = 0; g < 8 && g * W < items && tot < most; g++)
        {
            int cnt[16] = {0}, worst = 0;
            for (int l = 0; l < W && g * W + l < items; l++)
            {
                int c = ++cnt[mr_addr(k, s, g * W + l, col) % W];
                if (c > worst) worst = c;
            }
            tot += worst * k->radix[s] * (s > 0 && s < k->nstages - 1 ? 2 : 1);
        }
    }
    return tot;
}

static void mr_stride(fftz_pass_t *k, int colmap, int pad)
{
    const int W = k->dtype == 0 ? 16 : 8;
    int64_t s = mr_span(k, pad);
    /* neighbouring lines: an odd distance, or W / tpc apart where lanes run
     * across a power of two of lines */
    const int spread = colmap && k->tpc > 1 && k->tpc <= W && (k->tpc & (k->tpc - 1)) == 0;
    if (k->tpc > 1)
        while (spread ? (s % W) != W / k->tpc : (s & 1) == 0) s++;
    k->mr.pad = pad;
    k->sstride = (int32_t)s;
}

/* shared memory of a tile of c lines, without padding */
static int64_t mr_tile_bytes(fftz_pass_t *k, int colmap, int64_t c)
{
    k->tpc = (int32_t)c;
    mr_stride(k, colmap, 0);
    return fftz_pass_smem_bytes(k);
}

/* Fills k's mixed-radix launch shape (its lengths, strides, batch and flags are
 * set); want_tpc > 0 fixes the lines per CTA where they fit, threads > 0 the
 * block (the ragged executor's, whose tiles keep their size in small batches).
 * Returns 0, or -1 when the line does not fit cap bytes. */
int fz_mr_shape(fftz_pass_t *k, int want_tpc, int threads, int64_t cap)
{
    const int two = (k->flags & FFTZ_F_MID_TAB) != 0;
    const int colmap = k->in_mode == 1 || k->out_mode == 1;
    /* packed real lines: mirrored butterflies in the last (r2c) or first (c2r) stage */
    const int r2c = k->in_kind == FFTZ_IN_REAL_PAIRS, c2r = k->in_kind == FFTZ_IN_HERM_SEPARATE;
    /* row lines of up to 16 points in two stages where they factor: a thread that
     * holds a whole line reads it in steps of the line's length (measured on B200,
     * two stages against the former kernel: 6 x 300000 float 9 / 44 us, 12 19 / 48, 15
     * 26 / 52) */
    const int small = !colmap && !r2c && !c2r && k->n <= 16 && k->n >= 4 && k->n != 5 && k->n != 7 && k->n != 11 && k->n != 13;
    k->nstages = fz_mr_radices(k->n, two || small ? 2 : 1, r2c || c2r, k->radix, NULL);
    if (k->nstages <= 0) return -1;
    const int ps = r2c ? k->nstages - 1 : c2r ? 0 : -1; /* the paired stage */
    if (c2r)
        for (int s = 0; s < k->nstages / 2; s++)
        {
            const int32_t x = k->radix[s];
            k->radix[s] = k->radix[k->nstages - 1 - s];
            k->radix[k->nstages - 1 - s] = x;
        }
    k->variant = FFTZ_VAR_MR;
    k->mr.big = 0;
    int64_t M = k->n, B = 1;
    for (int s = 0; s < k->nstages; s++)
    {
        const int R = k->radix[s];
        if (R == 11 || R == 13) k->mr.big = 1;
        M /= R;
        fftz_mr_stage_t *st = &k->mr.st[s];
        st->r = R;
        st->m = (int32_t)M;
        st->nb = k->n / R;
        st->mg_nb = magic(st->nb);
        st->mg_m = magic(M);
        st->mg_r = magic(R);
        st->mg_b = magic(B);
        if (s > 0) B *= R;
    }
    k->tpc = 1;
    mr_stride(k, colmap, 0);
    const int tmax = fftz_mr_max_threads(k->dtype, k->mr.big);
    int64_t most = mr_lines(k, cap);
    if (most < 1) return -1;
    if (most > k->ntf) most = k->ntf;
    if (most > (threads ? FZ_RG_LINES : 256)) most = threads ? FZ_RG_LINES : 256;
    /* lines per CTA: about 4096 float / 2048 double points of row lines; whole
     * segments of neighbouring lines where lanes run across them. Of equal choices
     * the smaller tile (512-point double r2c rows x 262144: 2 lines 588, 4 521, 6 591,
     * 8 546 us). The executor's tiles, which wait on memory at their ends, are larger
     * (measured on B200, 4096 ragged transforms, forward: float 1536 points 888 us, 3072 839, 4096
     * 809, 6144 805; double 768 2124, 1536 1753, 2048 1459, 3072 1388, and with later
     * stage forms 2048 1298, 3072 1236, 4096 1187 us) */
    const int64_t pts = threads ? (k->dtype == 0 ? 6144 : 4096) : (k->dtype == 0 ? 4096 : 2048);
    int64_t lo = 1, hi = most;
    if (want_tpc > 0)
        lo = hi = want_tpc < most ? want_tpc : most;
    else if (colmap)
    {
        /* 8 neighbours (double lines above 440 points, whose 8 would leave fewer than
         * four CTAs an SM: 4), doubled while a tile stays small. Measured on B200, lines
         * a tile 4 / 6 / 8 / 12 / 16: 120000 x 64 double (375 and 320 points) 178 / 160 / 154 / 191 / 183 us, 60000 x 64 float (250 and
         * 240) 56 / 51 / 49 / 58 / 54, 1080-point float columns 66 / 56 / 51 / 56 / 51;
         * 65521 x 32 double (512-point rows of its middle pass) 161 with 4, 182 with 8.
         * Two sweeps of more than 1024 float points: 4 as well (convolutions of 2048 and
         * 4096 points x 4096 columns: 85 / 146 us with 4, 101 / 268 with the most that fit) */
        const int64_t seg = (k->dtype == 0 ? !two || k->n <= 1024 : k->n <= 440) ? 8 : 4, room = threads ? pts : pts / 2;
        lo = hi = seg < most ? seg : most;
        while (hi * 2 <= most && hi * 2 * k->n <= room && hi < 32) lo = hi = hi * 2;
        /* the executor's block is fixed: a few more columns where they fill it better */
        if (threads) hi = lo + lo / 2 <= most ? lo + lo / 2 : most;
    }
    else
    {
        /* fewer lines where whole CTAs would not give every SM two */
        while (hi > 1 && (hi * k->n > pts + pts / 2 || (threads == 0 && k->ntf / hi < 2 * 148))) hi--;
        lo = hi > 3 ? hi / 3 : 1;
    }
    /* `most` counts lines at the distance that a tile of one has; several are
     * further apart */
    while (hi > 1 && mr_tile_bytes(k, colmap, hi) > cap) hi--;
    if (lo > hi) lo = hi;
    if (colmap && !threads && want_tpc <= 0 && mr_tile_bytes(k, colmap, hi) > 114 * 1024)
    {
        /* Tiles that leave an SM one CTA. Columns that one round of CTAs can take: few a
         * tile, since nothing but latency counts then, a power of two of them (whole
         * sectors at the strided end). B200, columns a tile: float 5000 x 64 1 13.6, 5 30.7
         * us; x 300 4 18.8, 5 28.6; 9000 x 64 1 25.7, 3 43.7; double 4840 x 17 1 15.2, 2 18.6;
         * smaller tiles gain nothing (the passes of a 120000-point double line: 8 16.7, 4
         * 18.6). From four rounds on a power of two as well: float 5000 x 4096 4 158, 5 248
         * us; 7260 x 4096 2 303, 3 354; double 3630 x 4096 2 240, 3 262 */
        int64_t c = 1;
        while (c * 148 < k->ntf) c *= 2;
        if (c < hi)
            lo = hi = c;
        else if (k->ntf >= 4 * 148 * hi)
        {
            while (hi & (hi - 1)) hi &= hi - 1;
            lo = hi;
        }
    }
    double best = -1;
    int btpc = 1, bthr = 32;
    for (int64_t c = lo; c <= hi; c++)
    {
        const int64_t smem = mr_tile_bytes(k, colmap, c) + 1024;
        if (smem - 1024 > cap) continue;
        int64_t by_smem = (228 * 1024) / smem;
        if (by_smem > 24) by_smem = 24;
        /* a batch of one CTA an SM at most: the block that fills it alone. (Chosen as if
         * others ran beside it, blocks were small: B200, double 2197 points x 1 11.8 us,
         * 8.3 on the kernel before, float columns 2000 x 64 13.3.) */
        const int alone = !threads && (k->ntf + c - 1) / c <= 148;
        for (int t = threads ? threads : 64; t <= (threads ? threads : tmax); t += 32)
        {
            int64_t ctas = tmax / t;
            if (ctas > by_smem) ctas = by_smem;
            if (alone) ctas = 1;
            double used = 0, spent = 0;
            for (int s = 0; s < k->nstages; s++)
            {
                const int64_t nb = k->n / k->radix[s], items = c * (s == ps ? (nb + 1) / 2 : nb);
                const int w = mr_cost(k->radix[s]) * (s == ps ? 2 : 1);
                used += (double)items * w;
                spent += (double)((items + t - 1) / t * t) * w;
            }
            /* lanes at work, times warps in flight (half weight), times the
             * overlap of independent CTAs' phases */
            double occ = (double)(ctas * t) / tmax;
            double sc = used / spent * (0.4 + 0.6 * occ) * (ctas >= 4 ? 1.0 : ctas == 3 ? 0.98 : ctas == 2 ? 0.94 : 0.8);
            if (sc > best + 1e-9)
            {
                best = sc;
                btpc = (int)c;
                bthr = t;
            }
        }
    }
    k->tpc = btpc;
    k->threads = bthr;
    k->tpt = bthr / btpc > 0 ? bthr / btpc : 1;
    /* the digit-0 pad with the fewest bank conflicts that still fits */
    int bp = -1, bc = 0;
    for (int pad = 0; pad < (k->nstages > 1 ? 16 : 1); pad++)
    {
        mr_stride(k, colmap, pad);
        if (pad > 0 && fftz_pass_smem_bytes(k) > cap) break;
        const int c = mr_conflicts(k, bp < 0 ? 0x7fffffff : bc);
        if (bp < 0 || c < bc)
        {
            bp = pad;
            bc = c;
        }
    }
    mr_stride(k, colmap, bp);
    k->mr.mg_tpc = magic(k->tpc);
    if (ps >= 0) k->mr.mg_pair = magic((k->n / k->radix[ps] + 1) / 2);
    k->use_tma = 0;
    k->smem_tw = 0;
    return fftz_pass_smem_bytes(k) <= cap ? 0 : -1;
}

/* Mean gain of the radix-R butterfly less one: its constants (cos and sin of
 * 2 pi / R and its multiples) are rounded to the working precision, the same way
 * in every butterfly of every line, and the part of that error along the exact
 * transform, trace(F^H F~) / R^2 - 1, adds up over a line's stages (float 9 x 9 x 9 x 3:
 * -5e-8 of an error of 1.4e-7). Evaluated at 40 digits from the codelets' constants;
 * a composite's is the sum of its factors'. */
double fz_mr_gain(int dtype, int R)
{
    static const double g[2][17] = {
        {0, 0, 0, -5.98e-9, 0, 8.59e-9, -5.98e-9, -4.62e-9, -4.28e-9, -1.57e-8, 8.59e-9, -3.25e-9, -5.98e-9, 5.56e-10,
         -4.62e-9, 2.61e-9, -1.14e-8},
        {0, 0, 0, -1.93e-17, 0, -1.25e-18, -1.93e-17, -1.50e-18, 1.71e-17, -4.22e-17, -1.25e-18, -1.32e-17, -1.93e-17,
         -7.96e-18, -1.50e-18, -2.06e-17, 1.40e-17}};
    return R >= 0 && R <= 16 ? g[dtype == 0 ? 0 : 1][R] : 0;
}

/* Stage twiddles of a mixed-radix line: stage s multiplies by
 * W_{R_s M_s}^{k r} at [(k - 1) M_s + r], which is the Stockham table of the
 * reversed radix list. The table takes the butterflies' mean gain back: each of
 * its S - 1 products but the trivial ones by the same share (up to 64 points the
 * few roots' own rounding is what counts). Returns the blob offset, -1 on
 * allocation failure. */
int64_t fz_mr_twiddles(fz_blob *b, fftz_pass_t *k)
{
    int32_t rev[FFTZ_MR_STAGES] = {0}, off[FFTZ_MR_STAGES];
    const int S = k->nstages;
    for (int s = 0; s < S; s++) rev[s] = k->radix[S - 1 - s];
    double gain = 0, share = 0;
    for (int s = 0; s < S; s++)
    {
        gain += fz_mr_gain(k->dtype, k->radix[s]);
        if (s < S - 1) share += (1.0 - 1.0 / k->radix[s]) * (1.0 - 1.0 / k->mr.st[s].m);
    }
    const int64_t o = fz_stage_twiddles(b, k->dtype, k->n, S, rev, off, k->n > 64 ? -gain / share : 0);
    k->ntw = 1;
    for (int s = 0; s < S; s++) k->ntw += s < S - 1 ? (k->radix[s] - 1) * k->mr.st[s].m : 0;
    for (int s = 0; s < S; s++) k->mr.st[s].tw = k->tw_off[s] = off[S - 1 - s];
    return o;
}
