// CPU unit test of the quarter-wise K decode of csrc/khq_kdecode3.cuh (kq_open, kq_word, kq_word_dense, kq_word_slow):
// ternary and signed-code operand words against a plain per-dim decode, over words with more than eight outliers, rows
// with more than 50 outlier symbols and quarters with more than the window holds.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "khq_kdecode3.cuh"

int main(int argc, char** argv) {
    using namespace khq3;
    const double p_out = atof(argv[1]);
    std::mt19937 rng(977);
    long n_dense = 0, n_slow = 0, n_past = 0;
    for (int iter = 0; iter < 4000; ++iter) {
        uint32_t mask[16] = {0}, kp[40];
        for (uint32_t& v : kp) v = rng();
        const unsigned char* pb = reinterpret_cast<const unsigned char*>(kp);
        uint16_t t_want[256], c_want[256];
        uint32_t ord = 0;
        for (int d = 0; d < 256; ++d) {
            const double u = (rng() & 0xFFFFFF) / double(0x1000000);
            const uint32_t sym = u < p_out ? 3u : rng() % 3u;
            mask[d / 16] |= sym << (2 * (d % 16));
            t_want[d] = sym == 1 ? 0xBC00 : sym == 2 ? 0x3C00 : 0;
            c_want[d] = 0;
            if (sym == 3) {
                const bool in = ord < 50;
                const bool pos = in && ((pb[29 + ord / 8] >> (ord % 8)) & 1);
                t_want[d] = pos ? 0x3C00 : 0xBC00;
                c_want[d] = (pos ? 0 : 0x8000) | (in ? (pb[4 + ord / 2] >> (4 * (ord % 2))) & 15 : 0);
                n_past += !in;
                ++ord;
            }
        }
        uint32_t first = 0;
        for (int quarter = 0; quarter < 4; ++quarter) {
            uint32_t cnt = 0;
            for (int w = 0; w < 4; ++w) cnt += k3_count(mask[4 * quarter + w]);
            KQuarter q;
            kq_open(q, kp, first, cnt);
            uint32_t ob = first;
            for (int w = 0; w < 4; ++w) {
                const uint32_t word = mask[4 * quarter + w], n = k3_count(word);
                uint32_t t2[8], c2[8];
                if (cnt > KQ_MAX) {
                    kq_word_slow(word, ob, kp, t2, c2);
                    ++n_slow;
                } else if (n > 8) {
                    kq_word_dense(q, word, t2, c2);
                    ++n_dense;
                } else {
                    kq_word(q, word, n, t2, c2);
                }
                ob += n;
                for (int i = 0; i < 16; ++i) {
                    const int d = 64 * quarter + 16 * w + k3_dim_of(i);
                    const uint32_t t = (t2[i >> 1] >> (16 * (i & 1))) & 0xFFFF, c = (c2[i >> 1] >> (16 * (i & 1))) & 0xFFFF;
                    if (t != t_want[d] || (c != c_want[d] && ((c | c_want[d]) & 0x7FFF))) {  // -0 is 0
                        printf("iter %d dim %d: t %04x want %04x, c %04x want %04x\n", iter, d, t, t_want[d], c, c_want[d]);
                        return 1;
                    }
                }
            }
            first += cnt;
        }
    }
    printf("ok: %ld dense words, %ld words on the per-dim path, %ld entries past the format\n", n_dense, n_slow, n_past);
    return 0;
}
