// Host build of textscan.cuh's word-wise field functions for tests/test_textscan_cpu.py: reads one
// field per line from stdin as "<kind> <hex bytes>" (kind: i = integer, f = double, d = date), runs the
// word-wise function the scan kernels run first and the byte-wise one, and prints
// "<taken word-wise> <word-wise value> <byte-wise status> <byte-wise value>" (doubles as their bits;
// a value of 0 where the status carries none).
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "textscan.cuh"

static int hexval(char c) { return c <= '9' ? c - '0' : (c | 0x20) - 'a' + 10; }

int main() {
    char line[1 << 12];
    std::vector<char> buf;
    while (std::fgets(line, sizeof line, stdin)) {
        const char kind = line[0];
        buf.assign(32, 'x');  // what lies before a field is not part of it
        for (const char* p = line + 2; p[0] && p[0] != '\n' && p[1]; p += 2)
            buf.push_back((char)(hexval(p[0]) * 16 + hexval(p[1])));
        const long long n = (long long)buf.size() - 32;
        buf.resize(buf.size() + 16, '7');  // nor what lies after it
        const char* s = buf.data() + 32;
        bool fast = false;
        int slow = 0;
        long long fv = 0, sv = 0;
        unsigned w[4];
        const long long neg = n > 0 && s[0] == '-';
        if (kind == 'd') {
            int days = 0;
            std::memcpy(w, s, 12);
            if (n == 10) fast = ral_txw_date(w, &days);
            fv = days;
            slow = ral_tx_parse_date(s, 0, n, false, &sv);
        } else {
            std::memcpy(w, s + n - 16, 16);
            const bool fits = n <= 16 && n - neg > 0;
            if (kind == 'i') {
                if (fits) fast = n - neg <= 8 ? ral_txw_int8(w + 2, (unsigned)(n - neg), &fv) : ral_txw_int16(w, (unsigned)(n - neg), &fv);
                if (neg) fv = -fv;
                slow = ral_tx_parse_int(s, 0, n, &sv);
            } else {
                double a = 0, b = 0;
                if (fits) fast = ral_txw_double(w, (unsigned)(n - neg), &a);
                if (neg) a = -a;
                std::memcpy(&fv, &a, 8);
                slow = ral_tx_parse_double(s, 0, n, &b);
                std::memcpy(&sv, &b, 8);
            }
        }
        std::printf("%d %lld %d %lld\n", (int)fast, fast ? fv : 0ll, slow, slow == RAL_TX_OK ? sv : 0ll);
    }
    return 0;
}
