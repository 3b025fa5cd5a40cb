/* Roots of unity, stage twiddles, a forward FFT and the chirp spectrum for tables.c,
 * which includes this once for each REAL it forms tables in; FORM(name) is the
 * function's name there. */

/* All N roots exp(-2 pi i r / N), interleaved, by malloc (NULL on failure):
 * w_nl on the part of the circle that the reflections at N / 2, N / 4 and N / 8
 * leave (each where it divides N), mirrored to the rest. */
static REAL *FORM(roots)(int64_t N)
{
    REAL *w = (REAL *)malloc(sizeof(REAL) * 2 * (size_t)N);
    if (!w) return NULL;
    const int64_t half = N / 2, quarter = N % 2 == 0 ? N / 4 : half, eighth = N % 4 == 0 ? N / 8 : quarter;
    for (int64_t r = 0; r <= eighth; r++)
    {
        long double re, im;
        w_nl(r, N, &re, &im);
        w[2 * r] = (REAL)re;
        w[2 * r + 1] = (REAL)im;
    }
    if (N % 4 == 0) /* W^{N/4 - r} = -i conj(W^r) */
        for (int64_t r = eighth + 1; r <= N / 4; r++)
        {
            w[2 * r] = -w[2 * (N / 4 - r) + 1];
            w[2 * r + 1] = -w[2 * (N / 4 - r)];
        }
    if (N % 2 == 0) /* W^{N/2 - r} = -conj(W^r) */
        for (int64_t r = quarter + 1; r <= half; r++)
        {
            w[2 * r] = -w[2 * (half - r)];
            w[2 * r + 1] = w[2 * (half - r) + 1];
        }
    for (int64_t r = half + 1; r < N; r++) /* W^{N - r} = conj(W^r) */
    {
        w[2 * r] = w[2 * (N - r)];
        w[2 * r + 1] = -w[2 * (N - r) + 1];
    }
    return w;
}

/* Entries of a stage-twiddle table at off: every W_{Ns*R}^{k*r} is a root of order N,
 * the product of the radices; those but +-1 and +-i times 1 + gain. */
static int FORM(stage_entries)(fz_blob *b, int64_t off, int dtype, int nstages, const int32_t *radix,
                               const int32_t *tw_off, int64_t N, double gain)
{
    REAL *w = FORM(roots)(N);
    if (!w) return -1;
    for (int64_t r = 0; gain != 0 && r < N; r++)
        if (w[2 * r] != 0 && w[2 * r + 1] != 0)
        {
            w[2 * r] *= 1 + (REAL)gain;
            w[2 * r + 1] *= 1 + (REAL)gain;
        }
    int64_t ns = radix[0];
    for (int s = 1; s < nstages; s++)
    {
        const int64_t R = radix[s], step = N / (ns * R);
        for (int64_t r = 1; r < R; r++)
            for (int64_t k = 0; k < ns; k++)
                put_c(b, off, dtype, tw_off[s] + (r - 1) * ns + k, (double)w[2 * (k * r * step)],
                      (double)w[2 * (k * r * step) + 1]);
        ns *= R;
    }
    free(w);
    return 0;
}

/* Forward FFT, m a product of 2, 3, 5 and 7: Stockham stages of 4 and the prime
 * factors between x and a second buffer. w: roots of order m ws. Returns 0, or -1 on
 * allocation failure. */
static int FORM(host_fft)(REAL *x, int64_t m, const REAL *w, int64_t ws)
{
    REAL *y = (REAL *)malloc(sizeof(REAL) * 2 * (size_t)m);
    REAL *src = x, *dst = y;
    if (!y) return -1;
    int64_t n = m, st = 1; /* length still to transform, transforms side by side */
    while (n > 1)
    {
        const int p = n % 4 == 0 ? 4 : n % 2 == 0 ? 2 : n % 3 == 0 ? 3 : n % 5 == 0 ? 5 : 7;
        const int64_t h = n / p;
        REAL e[7][2]; /* W_p^j */
        for (int j = 0; j < p; j++)
        {
            e[j][0] = w[2 * (j * (m / p) * ws)];
            e[j][1] = w[2 * (j * (m / p) * ws) + 1];
        }
        for (int64_t k = 0; k < h; k++)
            for (int64_t q = 0; q < st; q++)
            {
                REAL v[7][2], o[7][2];
                for (int j = 0; j < p; j++)
                {
                    v[j][0] = src[2 * (q + st * (k + j * h))];
                    v[j][1] = src[2 * (q + st * (k + j * h)) + 1];
                }
                if (p == 4)
                {
                    const REAL ar = v[0][0] + v[2][0], ai = v[0][1] + v[2][1], br = v[0][0] - v[2][0],
                                 bi = v[0][1] - v[2][1], cr = v[1][0] + v[3][0], ci = v[1][1] + v[3][1],
                                 dr = v[1][0] - v[3][0], di = v[1][1] - v[3][1];
                    o[0][0] = ar + cr, o[0][1] = ai + ci, o[2][0] = ar - cr, o[2][1] = ai - ci;
                    o[1][0] = br + di, o[1][1] = bi - dr, o[3][0] = br - di, o[3][1] = bi + dr;
                }
                else
                    for (int r = 0; r < p; r++)
                    {
                        o[r][0] = v[0][0];
                        o[r][1] = v[0][1];
                        for (int j = 1, i = r; j < p; j++, i = i + r >= p ? i + r - p : i + r)
                        {
                            o[r][0] += v[j][0] * e[i][0] - v[j][1] * e[i][1];
                            o[r][1] += v[j][0] * e[i][1] + v[j][1] * e[i][0];
                        }
                    }
                for (int r = 0; r < p; r++) /* output r of the butterfly, times W_n^{k r} */
                {
                    const REAL *t = w + 2 * (k * r * st * ws);
                    REAL *d = dst + 2 * (q + st * (p * k + r));
                    d[0] = o[r][0] * t[0] - o[r][1] * t[1];
                    d[1] = o[r][0] * t[1] + o[r][1] * t[0];
                }
            }
        REAL *sw = src;
        src = dst;
        dst = sw;
        st *= p;
        n = h;
    }
    if (src != x) memcpy(x, src, sizeof(REAL) * 2 * (size_t)m);
    free(y);
    return 0;
}

/* The same of an even sequence, x_j = x_{m - j}, whose spectrum is even too: bins 2k
 * are the half-length transform of x_j + x_{j + m/2}, again even, bins 4k + 1 one of
 * a quarter of the length, and bin 4k + 3 is bin m - 4k - 3, one of those. Half the
 * work of host_fft. */
static int FORM(even_fft)(REAL *x, int64_t m, const REAL *w, int64_t ws)
{
    if (m % 4 != 0) return FORM(host_fft)(x, m, w, ws);
    const int64_t h = m / 2, q = m / 4;
    REAL *e = (REAL *)malloc(sizeof(REAL) * 2 * (size_t)(h + q)), *y = e + 2 * h;
    if (!e) return -1;
    for (int64_t j = 0; j < 2 * h; j++) e[j] = x[j] + x[j + 2 * h];
    for (int64_t j = 0; j < q; j++)
    {
        const REAL ar = x[2 * j] - x[2 * (j + h)], ai = x[2 * j + 1] - x[2 * (j + h) + 1];
        const REAL br = x[2 * (j + q)] - x[2 * (j + q + h)], bi = x[2 * (j + q) + 1] - x[2 * (j + q + h) + 1];
        const REAL re = ar + bi, im = ai - br, *t = w + 2 * (j * ws); /* a - i b */
        y[2 * j] = re * t[0] - im * t[1];
        y[2 * j + 1] = re * t[1] + im * t[0];
    }
    const int rc = FORM(even_fft)(e, h, w, 2 * ws) || FORM(host_fft)(y, q, w, 4 * ws) ? -1 : 0;
    for (int64_t k = 0; rc == 0 && k < q; k++)
        for (int c = 0; c < 2; c++)
        {
            x[2 * (4 * k) + c] = e[2 * (2 * k) + c];
            x[2 * (4 * k + 1) + c] = y[2 * k + c];
            x[2 * (4 * k + 2) + c] = e[2 * (2 * k + 1) + c];
            x[2 * (4 * k + 3) + c] = y[2 * (q - 1 - k) + c];
        }
    free(e);
    return rc;
}

/* c: the chirp c_j = exp(-i pi (j^2 mod 2n) / n) = W_{2n}^{j^2 mod 2n}, j < n
 * (core/common/bluestein_utils.c:88-159 keeps the square exact in integers); bb:
 * 1 / m times the m-point spectrum of conj(c_j) at j and m - j, zero between. */
static int FORM(chirp_spectrum)(int64_t n, int64_t m, double *c, double *bb)
{
    const int64_t n2 = 2 * n;
    REAL *w = FORM(roots)(n2), *x = (REAL *)calloc(2 * (size_t)m, sizeof(REAL));
    int rc = !w || !x ? -1 : 0;
    for (int64_t j = 0; rc == 0 && j < n; j++)
    {
        const int64_t sq = (int64_t)(((unsigned __int128)j * (unsigned __int128)j) % (unsigned __int128)n2);
        c[2 * j] = (double)w[2 * sq];
        c[2 * j + 1] = (double)w[2 * sq + 1];
        x[2 * j] = w[2 * sq];
        x[2 * j + 1] = -w[2 * sq + 1];
        if (j > 0)
        {
            x[2 * (m - j)] = w[2 * sq];
            x[2 * (m - j) + 1] = -w[2 * sq + 1];
        }
    }
    free(w);
    w = rc == 0 ? FORM(roots)(m) : NULL;
    rc = w ? FORM(even_fft)(x, m, w, 1) : -1;
    free(w);
    for (int64_t j = 0; rc == 0 && j < 2 * m; j++) bb[j] = (double)(x[j] / (REAL)m);
    free(x);
    return rc;
}
