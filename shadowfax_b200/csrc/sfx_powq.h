/*
 * sfx_powq: sfx_pow's value, bit for bit, at about a fifth of its cost, for
 * the plain-FP64 exact solver (host and device code).
 *
 * sfx_pow (sfx_pow.h) returns the correctly rounded power except within 2^-90
 * of a rounding boundary.  sfx_powq evaluates the power with table-driven
 * reductions, to about 2^-71 (1 + |y|): the logarithm's error is multiplied by
 * the exponent.  It rounds the value once, but only where no rounding boundary
 * lies within a margin of 2^-68 + |y| 2^-70 (Ziv's rounding test: A. Ziv, "Fast
 * evaluation of elementary mathematical functions with correctly rounded last
 * bit", ACM TOMS 17, 1991); there both routines return the same double.
 * Elsewhere (about 1 argument in 10^4 for |y| <= 5, 1 in 440 at |y| = 202 and
 * all above |y| = 2^17), outside x > 0 normal, and for |y ln x| >= 22, it calls
 * SFX_POWQ_RARE (sfx_pow, or the includer's out-of-line copy of it).
 *
 * Method (P. T. P. Tang, "Table-driven implementation of the logarithm
 * function", ACM TOMS 16, 1990, and "... of the exponential function", ACM
 * TOMS 15, 1989; the sums kept as unevaluated pairs):
 *   x = 2^e m, c ~ 1/m from the top 6 bits of m (64 entries of 8 bits),
 *   r = m c - 1 as a pair (|r| < 2^-6.6),
 *   ln x = e ln2 - ln c + r - r^2/2 + (r^3/3 - ... + r^11/11);
 *   t = y ln x;  k = nearest integer to 32 t / ln2,  r = t - k ln2/32,
 *   exp t = 2^(k div 32) 2^((k mod 32)/32) (1 + r + r^2/2 + ... + r^8/8!).
 * The tables hold -ln c and 2^(j/32) as pairs of doubles, evaluated in
 * 60-digit decimal arithmetic.
 */
#ifndef SFX_POWQ_H
#define SFX_POWQ_H

#include "sfx_pow.h"

#ifndef SFX_POWQ_RARE
#define SFX_POWQ_RARE sfx_pow
#endif

/* c, -ln c (high, low) for j = 0..63 */
#define SFX_POWQ_LOG_TABLE \
    0x1.fc00000000000p-1, 0x1.010157588de71p-7, 0x1.46662d417ced0p-62, \
    0x1.f400000000000p-1, 0x1.8492528c8cabfp-6, -0x1.d192d0619fa67p-60, \
    0x1.ec00000000000p-1, 0x1.466aed42de3eap-5, -0x1.cdd6f7f4a137ep-59, \
    0x1.e600000000000p-1, 0x1.aaef2d0fb10fcp-5, 0x1.a353bb42e0addp-61, \
    0x1.de00000000000p-1, 0x1.1973bd1465567p-4, -0x1.7558367a6acf6p-59, \
    0x1.d800000000000p-1, 0x1.4d3115d207eacp-4, 0x1.769f42c7842ccp-58, \
    0x1.d000000000000p-1, 0x1.9335e5d594989p-4, -0x1.478a85704ccb7p-58, \
    0x1.ca00000000000p-1, 0x1.c885801bc4b23p-4, 0x1.a38cb559a6706p-58, \
    0x1.c400000000000p-1, 0x1.fe89139dbd566p-4, -0x1.ac9f4215f9393p-58, \
    0x1.be00000000000p-1, 0x1.1aa2b7e23f72ap-3, -0x1.c6ef1d9b2ef7ep-59, \
    0x1.b800000000000p-1, 0x1.365fcb0159016p-3, 0x1.7d411a5b944adp-58, \
    0x1.b200000000000p-1, 0x1.527e5e4a1b58dp-3, -0x1.71a9682395bfdp-61, \
    0x1.ac00000000000p-1, 0x1.6f0128b756abcp-3, -0x1.8de59c21e166cp-57, \
    0x1.a600000000000p-1, 0x1.8beafeb38fe8cp-3, 0x1.55aa8b6997a40p-58, \
    0x1.a200000000000p-1, 0x1.9f6c407089664p-3, 0x1.35a19605e67efp-59, \
    0x1.9c00000000000p-1, 0x1.bd087383bd8adp-3, 0x1.dd355f6a516d7p-60, \
    0x1.9800000000000p-1, 0x1.d1037f2655e7bp-3, 0x1.60629242471a2p-57, \
    0x1.9200000000000p-1, 0x1.ef5ade4dcffe6p-3, -0x1.08ab2ddc708a0p-58, \
    0x1.8e00000000000p-1, 0x1.01eae5626c691p-2, -0x1.18290bd2932e2p-59, \
    0x1.8800000000000p-1, 0x1.1178e8227e47cp-2, -0x1.0e63a5f01c691p-57, \
    0x1.8400000000000p-1, 0x1.1bf99635a6b95p-2, -0x1.12aeb84249223p-57, \
    0x1.8000000000000p-1, 0x1.269621134db92p-2, 0x1.e0efadd9db02bp-56, \
    0x1.7a00000000000p-1, 0x1.36b6776be1117p-2, -0x1.324f0e883858ep-58, \
    0x1.7600000000000p-1, 0x1.419b423d5e8c7p-2, 0x1.0dbb243827392p-57, \
    0x1.7200000000000p-1, 0x1.4c9e09e172c3cp-2, -0x1.123615b147a5dp-58, \
    0x1.6e00000000000p-1, 0x1.57bf753c8d1fbp-2, -0x1.0908d15f88b63p-57, \
    0x1.6a00000000000p-1, 0x1.630030b3aac49p-2, 0x1.dc18ce51fff99p-57, \
    0x1.6600000000000p-1, 0x1.6e60ee6af1972p-2, 0x1.657c222d868cdp-58, \
    0x1.6200000000000p-1, 0x1.79e26687cfb3ep-2, -0x1.c168817443f22p-56, \
    0x1.5e00000000000p-1, 0x1.85855776dcbfbp-2, -0x1.486666443b153p-56, \
    0x1.5a00000000000p-1, 0x1.914a8635bf68ap-2, -0x1.ad4bb98c1f2c5p-56, \
    0x1.5800000000000p-1, 0x1.973a3431356aep-2, -0x1.89d2816cf838fp-57, \
    0x1.5400000000000p-1, 0x1.a33440224fa79p-2, -0x1.ba8062860ae23p-57, \
    0x1.5000000000000p-1, 0x1.af5295248cdd0p-2, 0x1.9d56c45dd3e86p-56, \
    0x1.4c00000000000p-1, 0x1.bb9611b80e2fbp-2, 0x1.6fd02999b21e1p-59, \
    0x1.4a00000000000p-1, 0x1.c1c60693fa39ep-2, -0x1.bfc00b8f3feaap-56, \
    0x1.4600000000000p-1, 0x1.ce42f18064743p-2, 0x1.0798270b29f39p-56, \
    0x1.4200000000000p-1, 0x1.dae75484c9616p-2, -0x1.0b5837185a661p-56, \
    0x1.4000000000000p-1, 0x1.e148a1a2726cep-2, -0x1.ac81cc8a4dfb8p-56, \
    0x1.3c00000000000p-1, 0x1.ee2a156b413e5p-2, -0x1.74b71fb5e57e3p-62, \
    0x1.3a00000000000p-1, 0x1.f4aa7ee03192dp-2, -0x1.0d487f5aba5e5p-57, \
    0x1.3600000000000p-1, 0x1.00e5ae5b207abp-1, 0x1.1713a36138e19p-57, \
    0x1.3400000000000p-1, 0x1.04360be7603adp-1, -0x1.17f9e54e78104p-57, \
    0x1.3000000000000p-1, 0x1.0ae76e2d054fap-1, 0x1.0d710fcfc4e0dp-55, \
    0x1.2e00000000000p-1, 0x1.0e4898611cce1p-1, 0x1.3300f002e836ep-55, \
    0x1.2c00000000000p-1, 0x1.11af823c75aa8p-1, -0x1.91eee7772c7c2p-55, \
    0x1.2800000000000p-1, 0x1.188ee40f23ca6p-1, 0x1.89df1568ca0b0p-55, \
    0x1.2600000000000p-1, 0x1.1c07849ae6007p-1, 0x1.59bddae1ccce2p-56, \
    0x1.2400000000000p-1, 0x1.1f8635fc61659p-1, -0x1.2164ff40e9817p-56, \
    0x1.2000000000000p-1, 0x1.269621134db92p-1, 0x1.e0efadd9db02bp-55, \
    0x1.1e00000000000p-1, 0x1.2a2786d0ec107p-1, -0x1.6a0c343be95dcp-56, \
    0x1.1c00000000000p-1, 0x1.2dbf557b0df43p-1, -0x1.b941ee770436bp-56, \
    0x1.1a00000000000p-1, 0x1.315da4434068bp-1, 0x1.6c3a5f12642c9p-57, \
    0x1.1600000000000p-1, 0x1.38ae2171976e7p-1, 0x1.21512aa596ea3p-55, \
    0x1.1400000000000p-1, 0x1.3c6080c36bfb5p-1, 0x1.1930603d87b6ep-56, \
    0x1.1200000000000p-1, 0x1.4019c2125ca93p-1, 0x1.86cf0f38b461ap-57, \
    0x1.1000000000000p-1, 0x1.43d9ff2f923c5p-1, -0x1.84f481051f71ap-56, \
    0x1.0e00000000000p-1, 0x1.47a1527e8a2d3p-1, 0x1.2541aca7d5844p-55, \
    0x1.0c00000000000p-1, 0x1.4b6fd6f970c1fp-1, 0x1.c457b531506f6p-55, \
    0x1.0a00000000000p-1, 0x1.4f45a835a4e19p-1, 0x1.d749362382a77p-56, \
    0x1.0800000000000p-1, 0x1.5322e26867857p-1, 0x1.988ba4aea614dp-56, \
    0x1.0600000000000p-1, 0x1.5707a26bb8c66p-1, 0x1.80bff3303dd48p-55, \
    0x1.0400000000000p-1, 0x1.5af405c3649e0p-1, -0x1.6714fbcd8135bp-55, \
    0x1.0200000000000p-1, 0x1.5ee82aa241920p-1, 0x1.1c066d235ee63p-56
/* 2^(j/32) (high, low) for j = 0..31 */
#define SFX_POWQ_EXP_TABLE \
    0x1.0000000000000p+0, 0x0.0p+0, \
    0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55, \
    0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54, \
    0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54, \
    0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55, \
    0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54, \
    0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54, \
    0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55, \
    0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55, \
    0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54, \
    0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55, \
    0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59, \
    0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56, \
    0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55, \
    0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54, \
    0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54, \
    0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54, \
    0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55, \
    0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55, \
    0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54, \
    0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54, \
    0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57, \
    0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56, \
    0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54, \
    0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54, \
    0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56, \
    0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55, \
    0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56, \
    0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55, \
    0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54, \
    0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54, \
    0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54

static const double sfx_powq_log_host[3 * 64] = {SFX_POWQ_LOG_TABLE};
static const double sfx_powq_exp_host[2 * 32] = {SFX_POWQ_EXP_TABLE};
#if defined(__CUDACC__)
static __device__ const double sfx_powq_log_dev[3 * 64] = {SFX_POWQ_LOG_TABLE};
static __device__ const double sfx_powq_exp_dev[2 * 32] = {SFX_POWQ_EXP_TABLE};
#endif

SFX_HD double sfx_powq_log_tab(int i) {
#if defined(__CUDA_ARCH__)
    return sfx_powq_log_dev[i];
#else
    return sfx_powq_log_host[i];
#endif
}

SFX_HD double sfx_powq_exp_tab(int i) {
#if defined(__CUDA_ARCH__)
    return sfx_powq_exp_dev[i];
#else
    return sfx_powq_exp_host[i];
#endif
}

/* ln x as a pair, absolute error below 2^-71 + 2^-100 |ln x| (the cubic term's
 * roundings, r^3 2^-52 and less, and the last sum's); 0: x is not a positive
 * normal number (the pair is then of no use).  No branches, here and
 * in sfx_powq_exp, so that two calls side by side overlap. */
SFX_HD int sfx_powq_log(double x, double* rh, double* rl) {
    const uint64_t u = sfx_d2u(x);
    const uint64_t ex = u >> 52; /* includes the sign bit */
    const double e = (double)((int)ex - 1023);
    const double m = sfx_u2d((u & 0x000fffffffffffffull) | 0x3ff0000000000000ull);
    const int j = 3 * (int)((u >> 46) & 63);
    const double c = sfx_powq_log_tab(j);
    const double ph = m * c;
    const double pl = sfx_fma(m, c, -ph);
    double r, s; /* r + s = m c - 1 (ph - 1 is exact) */
    sfx_fast_two_sum(ph - 1.0, pl, &r, &s);
    /* (r^3/3 - ... + r^11/11) / r^3 by pairs (Estrin): a chain of four */
    const double r2 = r * r, r4 = r2 * r2;
    const double q0 = sfx_fma(r, -1.0 / 4.0, 1.0 / 3.0), q2 = sfx_fma(r, -1.0 / 6.0, 1.0 / 5.0);
    const double q4 = sfx_fma(r, -1.0 / 8.0, 1.0 / 7.0), q6 = sfx_fma(r, -1.0 / 10.0, 1.0 / 9.0);
    const double q = sfx_fma(r4 * r4, 1.0 / 11.0,
                             sfx_fma(r4, sfx_fma(r2, q6, q4), sfx_fma(r2, q2, q0)));
    const double hr = -0.5 * r;
    const double qh = hr * r;
    const double ql = sfx_fma(hr, r, -qh);
    const double r3 = r * r2;
    /* the large parts exactly: e ln2_hi (42 significant bits) - ln c + r - r^2/2 */
    double h, e1, e2, e3;
    sfx_fast_two_sum(e * 0x1.62e42fefa3800p-1, sfx_powq_log_tab(j + 1), &h, &e1);
    sfx_two_sum(h, r, &h, &e2);
    sfx_two_sum(h, qh, &h, &e3);
    const double lo = sfx_fma(q, r3, ql) + sfx_fma(-r, s, s) +
                      sfx_fma(e, 0x1.ef35793c76730p-45, sfx_powq_log_tab(j + 2)) +
                      ((e1 + e2) + e3);
    sfx_fast_two_sum(h, lo, rh, rl); /* |lo| < 2^-21: off by 2^-75 where |h| is smaller */
    return ex - 1 < 0x7fe;
}

/* exp(th + tl) with th + tl = y ln x, rounded; 0: |th| >= 22 or NaN, or a
 * rounding boundary lies too near */
SFX_HD int sfx_powq_exp(double th, double tl, double y, double* out) {
    const double kd = (th * 0x1.71547652b82fep+5 + 0x1.8p52) - 0x1.8p52;
    const int in_range = (th < 0.0 ? -th : th) < 22.0; /* 0 for a NaN */
    const int k = in_range ? (int)kd : 0;
    const double a = th - kd * 0x1.62e42fefa3800p-6; /* exact */
    const double mh = kd * 0x1.ef35793c76730p-50;
    const double me = sfx_fma(kd, 0x1.ef35793c76730p-50, -mh);
    double r, s;
    sfx_fast_two_sum(a, -mh, &r, &s); /* |mh| < 2^-39: off by 2^-92 where |a| is smaller */
    sfx_fast_two_sum(r, s + (tl - me), &r, &s); /* tl is up to an ulp of th, not of r */
    const double r2 = r * r;
    const double q = sfx_fma(r2 * r2, sfx_fma(r, 1.0 / 40320.0, 1.0 / 5040.0),
                             sfx_fma(r2, sfx_fma(r, 1.0 / 720.0, 1.0 / 120.0),
                                     sfx_fma(r, 1.0 / 24.0, 1.0 / 6.0)));
    const double r2l = sfx_fma(r, r, -r2);
    /* exp(r + s) - 1 */
    double eh, el;
    sfx_fast_two_sum(r, 0.5 * r2, &eh, &el);
    el = el + (sfx_fma(r, s, s) + sfx_fma(q, r * r2, 0.5 * r2l));
    const int j = 2 * (k & 31);
    const double Th = sfx_powq_exp_tab(j), Tl = sfx_powq_exp_tab(j + 1);
    const double p = Th * eh;
    const double pl = sfx_fma(Th, eh, -p);
    double h, l;
    sfx_fast_two_sum(Th, p, &h, &l);
    l = l + (pl + sfx_fma(Th, el, sfx_fma(Tl, eh, Tl)));
    /* this function's error (below 2^-71) and |y| times the logarithm's */
    const double err = h * sfx_fma(y < 0.0 ? -y : y, 0x1p-70, 0x1p-68);
    const double up = h + (l + err), dn = h + (l - err);
    *out = up * sfx_u2d((uint64_t)((k >> 5) + 1023) << 52);
    return in_range & (up == dn);
}

SFX_HD double sfx_powq(double x, double y) {
    double lh, ll, r;
    if(sfx_powq_log(x, &lh, &ll)) {
        const double th = y * lh;
        const double tl = sfx_fma(y, lh, -th) + y * ll;
        if(sfx_powq_exp(th, tl, y, &r)) return r;
    }
    return SFX_POWQ_RARE(x, y);
}

#endif /* SFX_POWQ_H */
