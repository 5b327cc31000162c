// textscan.cuh — fields of delimited text rows parsed into column values (the scan side of a
// scan -> filter fusion).
//
// A table scan over a delimited text file (the reference's csv_parser, src/io/data_parser/
// CSVParser.cpp, which hands the bytes to cudf's CSV reader with '|' as the default delimiter, no
// header and blank lines skipped) turns each field into a value of the schema's dtype.  The rules
// here, shared by the GPU scan kernel and the host tests:
//
// * a field is the bytes between two delimiters (or a row's ends); spaces around it are ignored;
//   an empty field, or one that does not read as the dtype, is null;
// * integers: an optional sign and decimal digits, accumulated modulo 2^64 and narrowed to the
//   column's width by two's complement truncation;
// * floating point: an optional sign, digits with an optional decimal point, an optional exponent
//   (e or E, optional sign, up to five digits); the value is the decimal number rounded to the
//   nearest double (ties to even), then to float for FLOAT32 columns.  It is computed exactly
//   when the significand has at most 19 digits and either fits in 53 bits with a power of ten
//   |e| <= 22 (one correctly rounded multiply or divide of two exact doubles, Clinger's fast
//   path) or is small enough to absorb the excess power of ten; other values are refused (the
//   scan reports an error rather than round them differently);
// * dates: YYYY-MM-DD, years 0001-9999 (DATE32: days since 1970-01-01; DATE64: milliseconds),
//   and for DATE64 optionally a time HH:MM:SS after a space or 'T'; proleptic Gregorian, UTC.
//
// The file compiles as CUDA device code (the NVRTC prelude) and as plain C++ on the host, where
// the tests compare every function with the host's own conversions.
#ifndef RAL_TEXTSCAN_CUH_
#define RAL_TEXTSCAN_CUH_

#if defined(__CUDACC__) || defined(__CUDACC_RTC__)
#define RAL_TX __host__ __device__ __forceinline__
#else
#define RAL_TX static inline
#endif

// field validity: a value, a null, or a value this scan refuses to round
#define RAL_TX_NULL 0
#define RAL_TX_OK 1
#define RAL_TX_REFUSED 2

RAL_TX bool ral_tx_digit(unsigned char c) { return c >= '0' && c <= '9'; }

// [p, e) without the spaces at either end
RAL_TX void ral_tx_trim(const char* s, long long& p, long long& e) {
    while (p < e && s[p] == ' ') ++p;
    while (e > p && s[e - 1] == ' ') --e;
}

RAL_TX int ral_tx_parse_int(const char* s, long long p, long long e, long long* out) {
    ral_tx_trim(s, p, e);
    if (p >= e) return RAL_TX_NULL;
    bool neg = false;
    if (s[p] == '+' || s[p] == '-') {
        neg = s[p] == '-';
        ++p;
    }
    if (p >= e) return RAL_TX_NULL;
    unsigned long long v = 0;
    for (; p < e; ++p) {
        const unsigned char c = (unsigned char)s[p];
        if (!ral_tx_digit(c)) return RAL_TX_NULL;
        v = v * 10ull + (unsigned long long)(c - '0');
    }
    *out = (long long)(neg ? 0ull - v : v);
    return RAL_TX_OK;
}

// 10^k for k <= 22: every one is an exact double
RAL_TX double ral_tx_pow10(int k) {
    double r = 1.0;
    double b = 10.0;
    while (k) {  // exact: every partial product is a power of ten below 2^53 * 2^k
        if (k & 1) r *= b;
        b *= b;
        k >>= 1;
    }
    return r;
}

RAL_TX double ral_tx_mul(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
RAL_TX double ral_tx_div(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
}

RAL_TX int ral_tx_parse_double(const char* s, long long p, long long e, double* out) {
    ral_tx_trim(s, p, e);
    if (p >= e) return RAL_TX_NULL;
    bool neg = false;
    if (s[p] == '+' || s[p] == '-') {
        neg = s[p] == '-';
        ++p;
    }
    unsigned long long m = 0;
    int sig = 0;         // significant digits taken into m
    int e10 = 0;         // decimal exponent of m
    int digits = 0;      // digits seen in the significand
    bool dot = false;
    for (; p < e; ++p) {
        const unsigned char c = (unsigned char)s[p];
        if (c == '.') {
            if (dot) return RAL_TX_NULL;
            dot = true;
            continue;
        }
        if (!ral_tx_digit(c)) break;
        ++digits;
        if (m == 0 && c == '0') {  // a leading zero: only moves the exponent after the point
            if (dot) --e10;
            continue;
        }
        if (sig == 19) {  // a 20th significant digit: beyond the exact range unless it is zero
            if (c != '0') return RAL_TX_REFUSED;
            if (!dot) ++e10;
            continue;
        }
        m = m * 10ull + (unsigned long long)(c - '0');
        ++sig;
        if (dot) --e10;
    }
    if (digits == 0) return RAL_TX_NULL;
    if (p < e) {
        const unsigned char c = (unsigned char)s[p];
        if (c != 'e' && c != 'E') return RAL_TX_NULL;
        ++p;
        bool eneg = false;
        if (p < e && (s[p] == '+' || s[p] == '-')) {
            eneg = s[p] == '-';
            ++p;
        }
        if (p >= e) return RAL_TX_NULL;
        int x = 0, nd = 0;
        for (; p < e; ++p) {
            const unsigned char d = (unsigned char)s[p];
            if (!ral_tx_digit(d)) return RAL_TX_NULL;
            if (++nd > 5) return RAL_TX_REFUSED;
            x = x * 10 + (d - '0');
        }
        e10 += eneg ? -x : x;
    }
    double v;
    if (m == 0) {
        v = 0.0;
    } else {
        const unsigned long long two53 = 1ull << 53;
        if (e10 > 22 && m <= two53) {
            // absorb the excess power of ten into the significand while it stays exact
            while (e10 > 22 && m <= two53 / 10ull) {
                m *= 10ull;
                --e10;
            }
        }
        if (m > two53 || e10 > 22 || e10 < -22) return RAL_TX_REFUSED;
        const double dm = (double)m;  // exact: m <= 2^53
        v = e10 >= 0 ? ral_tx_mul(dm, ral_tx_pow10(e10)) : ral_tx_div(dm, ral_tx_pow10(-e10));
    }
    *out = neg ? -v : v;
    return RAL_TX_OK;
}

// Days from 1970-01-01 of a proleptic Gregorian date (the public days-from-civil algorithm: a
// year starting in March, 400-year eras of 146097 days).
RAL_TX long long ral_tx_days_from_civil(long long y, unsigned m, unsigned d) {
    y -= m <= 2 ? 1 : 0;
    const long long era = (y >= 0 ? y : y - 399) / 400;
    const unsigned yoe = (unsigned)(y - era * 400);
    const unsigned doy = (153u * (m + (m > 2 ? -3 : 9)) + 2u) / 5u + d - 1u;
    const unsigned doe = yoe * 365u + yoe / 4u - yoe / 100u + doy;
    return era * 146097ll + (long long)doe - 719468ll;
}

RAL_TX bool ral_tx_num(const char* s, long long p, int n, unsigned* out) {
    unsigned v = 0;
    for (int i = 0; i < n; ++i) {
        const unsigned char c = (unsigned char)s[p + i];
        if (!ral_tx_digit(c)) return false;
        v = v * 10u + (unsigned)(c - '0');
    }
    *out = v;
    return true;
}

// YYYY-MM-DD, and for with_time HH:MM:SS after ' ' or 'T'; *out = days, or milliseconds when
// with_time is set (the time optional).
RAL_TX int ral_tx_parse_date(const char* s, long long p, long long e, bool with_time, long long* out) {
    ral_tx_trim(s, p, e);
    if (p >= e) return RAL_TX_NULL;
    const long long n = e - p;
    if (n < 10 || s[p + 4] != '-' || s[p + 7] != '-') return RAL_TX_NULL;
    unsigned y, mo, d;
    if (!ral_tx_num(s, p, 4, &y) || !ral_tx_num(s, p + 5, 2, &mo) || !ral_tx_num(s, p + 8, 2, &d)) return RAL_TX_NULL;
    if (y < 1 || mo < 1 || mo > 12 || d < 1) return RAL_TX_NULL;  // years 0001-9999
    const bool leap = (y % 4u == 0u && y % 100u != 0u) || y % 400u == 0u;
    const unsigned mdays = mo == 2 ? (leap ? 29u : 28u) : ((mo == 4 || mo == 6 || mo == 9 || mo == 11) ? 30u : 31u);
    if (d > mdays) return RAL_TX_NULL;
    const long long days = ral_tx_days_from_civil((long long)y, mo, d);
    if (!with_time) {
        if (n != 10) return RAL_TX_NULL;
        *out = days;
        return RAL_TX_OK;
    }
    long long secs = 0;
    if (n != 10) {
        if (n != 19 || (s[p + 10] != ' ' && s[p + 10] != 'T') || s[p + 13] != ':' || s[p + 16] != ':')
            return RAL_TX_NULL;
        unsigned h, mi, se;
        if (!ral_tx_num(s, p + 11, 2, &h) || !ral_tx_num(s, p + 14, 2, &mi) || !ral_tx_num(s, p + 17, 2, &se))
            return RAL_TX_NULL;
        if (h > 23 || mi > 59 || se > 59) return RAL_TX_NULL;
        secs = (long long)h * 3600 + (long long)mi * 60 + (long long)se;
    }
    *out = (days * 86400ll + secs) * 1000ll;
    return RAL_TX_OK;
}

// ---- fields read as words ----------------------------------------------------------------------
// The common shapes of a field, read 4 bytes at a time instead of byte by byte and without branches: a
// number of at most 16 characters arrives in little-endian words aligned to its END (the last
// character is the top byte of the last word; bytes before the field's n are ignored), a date in three
// words aligned to its start.  Each function returns true with what the byte-wise function above gives
// for the same characters, or false, after which the caller runs the byte-wise one: signs other than the
// leading '-' the caller strips, spaces, exponents, 29 February, more characters and whatever does not
// read as the dtype.

// a.lo16 * b.byte0 + a.hi16 * b.byte1 + c / the same with b's bytes 2 and 3
RAL_TX unsigned ral_txw_dp2_lo(unsigned a, unsigned b, unsigned c) {
#if defined(__CUDA_ARCH__)
    unsigned d;
    asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
#else
    return (a & 0xffffu) * (b & 0xffu) + (a >> 16) * ((b >> 8) & 0xffu) + c;
#endif
}
RAL_TX unsigned ral_txw_dp2_hi(unsigned a, unsigned b, unsigned c) {
#if defined(__CUDA_ARCH__)
    unsigned d;
    asm("dp2a.hi.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
#else
    return (a & 0xffffu) * ((b >> 16) & 0xffu) + (a >> 16) * (b >> 24) + c;
#endif
}
// four digit values (0 .. 9 a byte, the first character lowest) as a number
RAL_TX unsigned ral_txw_dec4(unsigned x) {
    return ral_txw_dp2_lo(0x006403e8u, x, ral_txw_dp2_hi(0x0001000au, x, 0u));
}
RAL_TX unsigned ral_txw_dec8(unsigned long long x) {
    return ral_txw_dec4((unsigned)x) * 10000u + ral_txw_dec4((unsigned)(x >> 32));
}
// nonzero when a byte of x (characters ^ '0') is not 0 .. 9; a byte that carries into the next one
// is itself flagged
RAL_TX unsigned ral_txw_nondigit(unsigned x) { return (x | (x + 0x06060606u)) & 0xf0f0f0f0u; }
// 0x80 in each byte of x that is zero
RAL_TX unsigned ral_txw_zero_bytes(unsigned x) { return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u; }

RAL_TX unsigned ral_txw_ctz32(unsigned x) {
#if defined(__CUDA_ARCH__)
    return (unsigned)__ffs((int)x) - 1u;
#else
    return (unsigned)__builtin_ctz(x);
#endif
}

// bit k: the flag (0x80) of byte k of z0, z1, z2, z3
RAL_TX unsigned ral_txw_flags16(unsigned z0, unsigned z1, unsigned z2, unsigned z3) {
#if defined(__CUDA_ARCH__)
    unsigned lo = 0, hi = 0;  // 128 times the bits
    asm("dp4a.u32.u32 %0, %1, %2, %0;" : "+r"(lo) : "r"(z0), "r"(0x08040201u));
    asm("dp4a.u32.u32 %0, %1, %2, %0;" : "+r"(lo) : "r"(z1), "r"(0x80402010u));
    asm("dp4a.u32.u32 %0, %1, %2, %0;" : "+r"(hi) : "r"(z2), "r"(0x08040201u));
    asm("dp4a.u32.u32 %0, %1, %2, %0;" : "+r"(hi) : "r"(z3), "r"(0x80402010u));
    return (lo >> 7) | (hi << 1);
#else
    const unsigned z[4] = {z0, z1, z2, z3};
    unsigned r = 0;
    for (int k = 0; k < 16; ++k) r |= ((z[k >> 2] >> (8 * (k & 3) + 7)) & 1u) << k;
    return r;
#endif
}

// the last n (1 .. 8) of eight bytes, the others zero; any n stays defined
RAL_TX unsigned long long ral_txw_last(unsigned long long x, unsigned n) { return x & (~0ull << ((64u - 8u * n) & 63u)); }

// n (1 .. 8) digits in w[0..1]
RAL_TX bool ral_txw_int8(const unsigned* w, unsigned n, long long* out) {
    const unsigned long long x = ral_txw_last(((unsigned long long)w[1] << 32 | w[0]) ^ 0x3030303030303030ull, n);
    *out = (long long)ral_txw_dec8(x);
    return (n - 1u < 8u) & ((ral_txw_nondigit((unsigned)x) | ral_txw_nondigit((unsigned)(x >> 32))) == 0u);
}
// n (9 .. 16) digits in w[0..3]
RAL_TX bool ral_txw_int16(const unsigned* w, unsigned n, long long* out) {
    const unsigned long long hi = ((unsigned long long)w[3] << 32 | w[2]) ^ 0x3030303030303030ull;
    const unsigned long long lo = ral_txw_last(((unsigned long long)w[1] << 32 | w[0]) ^ 0x3030303030303030ull, n - 8u);
    *out = (long long)((unsigned long long)ral_txw_dec8(lo) * 100000000ull + ral_txw_dec8(hi));
    return (n - 9u < 8u) & ((ral_txw_nondigit((unsigned)hi) | ral_txw_nondigit((unsigned)(hi >> 32)) |
                             ral_txw_nondigit((unsigned)lo) | ral_txw_nondigit((unsigned)(lo >> 32))) == 0u);
}

// 1 / 10^f as the sum of two doubles, f = 0 .. 15
#if defined(__CUDACC_RTC__) || defined(__CUDACC__)
#define RAL_TX_TABLE static __constant__
#else
#define RAL_TX_TABLE static const
#endif
RAL_TX_TABLE double ral_txw_inv_hi[16] = {
    1e-0, 1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12, 1e-13, 1e-14, 1e-15};
RAL_TX_TABLE double ral_txw_inv_lo[16] = {
    0x0.0p+0, -0x1.999999999999ap-58, -0x1.eb851eb851eb8p-63, -0x1.89374bc6a7efap-66, -0x1.6a161e4f765fep-68,
    -0x1.ee78183f91e64p-71, 0x1.b5a63f9a49c2cp-75, 0x1.5e1e99483b023p-78, -0x1.03023df2d4c94p-82,
    -0x1.34674bfabb83bp-84, -0x1.20a5465df8d2cp-88, 0x1.7f7bc7b4d28aap-91, 0x1.97f27f0f6e886p-96,
    -0x1.ecd79a5a0df95p-99, 0x1.ea70909833de7p-107, -0x1.937831647f5a0p-104};

RAL_TX double ral_txw_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#else
    return __builtin_fma(a, b, c);
#endif
}

// A number of 1 .. 16 characters: digits with at most one point.  The value is m / 10^f rounded once, with
// m < 2^52 and f <= 15, as fma(m, yh, m * yl) where yh + yl is 10^-f to about 2^-106: the sum before
// its one rounding is within 2^-104 of m / 10^f relatively, and m / 10^f is either a double or
// further than 2^-54 / 5^f > 2^-90 from every midpoint of two doubles (the nearest such fractions
// differ by at least 1 / (5^f 2^j)), so the rounding is that of the exact quotient -- the value of
// the correctly rounded division.  Three FP64 instructions (with the exact conversion of m) in
// place of a division.
RAL_TX double ral_txw_scaled(unsigned long long m, unsigned f) {
#if defined(__CUDA_ARCH__)
    // m < 2^52 as the fraction of 2^52 + m: the subtraction is exact
    const double a = __dsub_rn(__longlong_as_double((long long)(0x4330000000000000ull | m)), 4503599627370496.0);
#else
    const double a = (double)(long long)m;
#endif
    return ral_txw_fma(a, ral_txw_inv_hi[f], ral_tx_mul(a, ral_txw_inv_lo[f]));
}
// n (1 .. 8) characters in w[0..1]: the digits before the point move up by its byte.  Half of the 16
// characters' instructions: a scan of 20M lines whose condition reads two such fields 836 -> 799 us.
RAL_TX bool ral_txw_double8(const unsigned* w, unsigned n, double* out) {
    const unsigned long long x = ral_txw_last(((unsigned long long)w[1] << 32 | w[0]) ^ 0x3030303030303030ull, n);
    const unsigned z0 = ral_txw_zero_bytes((unsigned)x ^ 0x1e1e1e1eu), z1 = ral_txw_zero_bytes((unsigned)(x >> 32) ^ 0x1e1e1e1eu);
    const unsigned long long z = (unsigned long long)z1 << 32 | z0;
    // the bytes up to the first point and its own; a second one stays and is no digit
    const unsigned long long upto = z ? z ^ (z - 1ull) : 0ull;
    const unsigned long long y = ((x << 8) & upto) | (x & ~upto);
    const unsigned f = (z0 ? 7u : 3u) - (ral_txw_ctz32(z0 ? z0 : z1 | 0x80000000u) >> 3);
    *out = ral_txw_scaled(ral_txw_dec8(y), z ? f : 0u);
    return (n - 1u < 8u) & ((ral_txw_nondigit((unsigned)y) | ral_txw_nondigit((unsigned)(y >> 32))) == 0u) &
           (n > (z ? 1u : 0u));
}
// n (9 .. 16) characters in w[0..3]
RAL_TX bool ral_txw_double16(const unsigned* w, unsigned n, double* out) {
    const unsigned long long hi = ((unsigned long long)w[3] << 32 | w[2]) ^ 0x3030303030303030ull;
    const unsigned long long lo = ral_txw_last(((unsigned long long)w[1] << 32 | w[0]) ^ 0x3030303030303030ull, n - 8u);
    unsigned x0 = (unsigned)lo, x1 = (unsigned)(lo >> 32), x2 = (unsigned)hi, x3 = (unsigned)(hi >> 32);
    // 0x80 at each point ('.' ^ '0' = 0x1e), which then reads as a zero digit
    const unsigned z0 = ral_txw_zero_bytes(x0 ^ 0x1e1e1e1eu), z1 = ral_txw_zero_bytes(x1 ^ 0x1e1e1e1eu);
    const unsigned z2 = ral_txw_zero_bytes(x2 ^ 0x1e1e1e1eu), z3 = ral_txw_zero_bytes(x3 ^ 0x1e1e1e1eu);
    const unsigned points = ral_txw_flags16(z0, z1, z2, z3);  // bit k: byte k
    x0 &= ~((z0 >> 2) - (z0 >> 7));
    x1 &= ~((z1 >> 2) - (z1 >> 7));
    x2 &= ~((z2 >> 2) - (z2 >> 7));
    x3 &= ~((z3 >> 2) - (z3 >> 7));
    const unsigned bad = ral_txw_nondigit(x0) | ral_txw_nondigit(x1) | ral_txw_nondigit(x2) | ral_txw_nondigit(x3) |
                         (points & (points - 1u));
    const unsigned vl = ral_txw_dec4(x0) * 10000u + ral_txw_dec4(x1), vh = ral_txw_dec4(x2) * 10000u + ral_txw_dec4(x3);
    const unsigned long long v = (unsigned long long)vl * 100000000ull + vh;
    // with a point v is the whole part times 10^(f + 1) plus the fraction B: (v - B) / 10 + B has the
    // point out (an exact division: by 2, then times the inverse of 5 modulo 2^64); without one B = v
    const unsigned f = points ? 15u - ral_txw_ctz32(points) : 0u;
    unsigned long long B = ral_txw_dec8(((unsigned long long)x3 << 32 | x2) & ((~0ull << 8) << ((56u - 8u * f) & 63u)));
    if (f >= 8u) B = (unsigned long long)ral_txw_dec8(((unsigned long long)x1 << 32 | x0) & ((~0ull << 8) << (120u - 8u * f))) * 100000000ull + vh;
    if (!points) B = v;
    const unsigned long long m = ((v - B) >> 1) * 0xcccccccccccccccdull + B;
    *out = ral_txw_scaled(m, f);
    return (n - 9u < 8u) & (bad == 0u) & ((m >> 52) == 0ull);
}
// n (1 .. 16) characters in w[0..3], w[0..1] only read for n > 8
RAL_TX bool ral_txw_double(const unsigned* w, unsigned n, double* out) {
    bool ok = ral_txw_double8(w + 2, n, out);
    if (n > 8u) ok = ral_txw_double16(w, n, out);
    return ok;
}

// YYYY-MM-DD in three words aligned to its start (the bytes after the tenth are ignored), 29 February left out: days since
// 1970-01-01 in 32-bit arithmetic
RAL_TX bool ral_txw_date(const unsigned* w, int* days) {
    const unsigned yx = w[0] ^ 0x30303030u;
    const unsigned mx = w[1] ^ 0x2d30302du;  // "-MM-"
    const unsigned dx = (w[2] ^ 0x3030u) & 0xffffu;
    const unsigned bad = (mx & 0xff0000ffu) | ral_txw_nondigit(yx) | ral_txw_nondigit(mx & 0x00ffff00u) | ral_txw_nondigit(dx);
    const unsigned y = ral_txw_dec4(yx);
    const unsigned mo = ((mx >> 8) & 0xffu) * 10u + ((mx >> 16) & 0xffu);
    const unsigned d = (dx & 0xffu) * 10u + (dx >> 8);
    // 30 or 31 days by the month's parity, which turns after July; 28 in February
    const unsigned most = mo == 2u ? 28u : 30u + ((mo + (mo >> 3)) & 1u);
    // a year starting in March: the days before it, then those of its months
    const unsigned yy = mo <= 2u ? y - 1u : y;
    const unsigned cc = yy / 100u;
    const unsigned doy = (153u * (mo > 2u ? mo - 3u : mo + 9u) + 2u) / 5u + d - 1u;
    *days = (int)(yy * 365u + (yy >> 2) - cc + (cc >> 2) + doy) - 719468;
    return (bad == 0u) & (y >= 1u) & (mo - 1u < 12u) & (d - 1u < most);
}

#if defined(__CUDACC_RTC__)
// ---- the scan kernels' views of staged text ------------------------------------------------------
// A warp holds text in shared memory as 32-bit words and one bit per byte that is set where the byte
// is the delimiter.  Byte positions are 32-bit numbers; kMask (words) wraps them into a ring, or is
// ~0 for an area addressed directly (which has 16 bytes to spare at both ends: a field's words may
// begin before it and end after it).

// One bit per byte of the 16 in v that equals c4's (c4: one byte four times).
__device__ __forceinline__ unsigned ral_txv_eq16(const uint4& v, unsigned c4) {
    return ral_txw_flags16(ral_txw_zero_bytes(v.x ^ c4), ral_txw_zero_bytes(v.y ^ c4), ral_txw_zero_bytes(v.z ^ c4),
                           ral_txw_zero_bytes(v.w ^ c4));
}

// The 16 bytes at p + at (a 16-byte aligned address), bytes outside [lo, hi) read as zero.
static __device__ __noinline__ uint4 ral_txv_edge16(const char* p, unsigned at, unsigned lo, unsigned hi) {
    unsigned w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (at + k >= lo && at + k < hi) w[k >> 2] |= (unsigned)(unsigned char)p[at + k] << (8 * (k & 3));
    return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint4 ral_txv_load16(const char* p, unsigned at, unsigned lo, unsigned hi) {
    if (at >= lo && at + 16u <= hi) return *reinterpret_cast<const uint4*>(p + at);
    if (at >= hi) return make_uint4(0u, 0u, 0u, 0u);
    return ral_txv_edge16(p, at, lo, hi);
}

template <unsigned kMask>
__device__ __forceinline__ unsigned ral_txv_byte(const unsigned* t, unsigned p) {
    return reinterpret_cast<const unsigned char*>(t)[p & (kMask * 4u + 3u)];
}

// N words of text from position p on
template <unsigned kMask, int N>
__device__ __forceinline__ void ral_txv_words(const unsigned* t, unsigned p, unsigned* w) {
    const unsigned i = p >> 2, s = 8u * (p & 3u);
    unsigned a = t[i & kMask];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned b = t[(i + k + 1u) & kMask];
        w[k] = __funnelshift_r(a, b, s);
        a = b;
    }
}

// the byte-wise functions, out of line: a field the word-wise ones leave (p: its first byte in global
// memory); the value as its 64 bits
struct ral_tx_result {
    long long v;
    int st;
};
static __device__ __noinline__ ral_tx_result ral_txv_slow_int(const char* p, long long n) {
    ral_tx_result r{0, 0};
    r.st = ral_tx_parse_int(p, 0, n, &r.v);
    return r;
}
static __device__ __noinline__ ral_tx_result ral_txv_slow_double(const char* p, long long n) {
    double d = 0.0;
    const int st = ral_tx_parse_double(p, 0, n, &d);
    return ral_tx_result{__double_as_longlong(d), st};
}
static __device__ __noinline__ ral_tx_result ral_txv_slow_date(const char* p, long long n, bool with_time) {
    ral_tx_result r{0, 0};
    r.st = ral_tx_parse_date(p, 0, n, with_time, &r.v);
    return r;
}

// The field at positions [fs, fe) of the staged text (fs < fe), word-wise.
template <unsigned kMask>
__device__ __forceinline__ bool ral_txv_int(const unsigned* t, unsigned fs, unsigned fe, long long* out) {
    const unsigned neg = ral_txv_byte<kMask>(t, fs) == '-' ? 1u : 0u, n = fe - fs - neg;
    unsigned w[4];
    ral_txv_words<kMask, 2>(t, fe - 8u, w);
    long long v;
    bool ok = ral_txw_int8(w, n, &v);
    if (n - 9u < 8u) {
        ral_txv_words<kMask, 4>(t, fe - 16u, w);
        ok = ral_txw_int16(w, n, &v);
    }
    *out = neg ? -v : v;
    return ok;
}
template <unsigned kMask>
__device__ __forceinline__ bool ral_txv_double(const unsigned* t, unsigned fs, unsigned fe, double* out) {
    const unsigned neg = ral_txv_byte<kMask>(t, fs) == '-' ? 1u : 0u;
    const unsigned n = fe - fs - neg;
    unsigned w[4] = {0u, 0u, 0u, 0u};
    ral_txv_words<kMask, 2>(t, fe - 8u, w + 2);
    if (n > 8u) ral_txv_words<kMask, 2>(t, fe - 16u, w);
    double v;
    const bool ok = ral_txw_double(w, n, &v);
    *out = __longlong_as_double(__double_as_longlong(v) ^ (long long)((unsigned long long)neg << 63));
    return ok;
}
template <unsigned kMask>
__device__ __forceinline__ bool ral_txv_date(const unsigned* t, unsigned fs, unsigned fe, bool with_time, long long* out) {
    unsigned w[3];
    ral_txv_words<kMask, 3>(t, fs, w);
    int days;
    const bool ok = ral_txw_date(w, &days);
    *out = with_time ? (long long)days * 86400000ll : (long long)days;
    return ok & (fe - fs == 10u);
}
#endif  // __CUDACC_RTC__

#endif  // RAL_TEXTSCAN_CUH_
