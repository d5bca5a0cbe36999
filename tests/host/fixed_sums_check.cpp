// The resident PCG's fixed-point sums (lightfem_gb300/csrc/cg_fixed.hpp) as its CTAs form
// them, on the host, for shares read from a file.
//
//   fixed_sums_check <in file> <out file>
//   in file:  int64 cases, then per case int64 mixed, CTAs, threads, double previous total,
//             double shares[CTAs][threads] (mixed: float hi and lo in place of a double)
//   out file: per case double accepted (0 or 1), limbs overflowed (0 or 1), total's high and low parts
#include "../../lightfem_gb300/csrc/cg_fixed.hpp"

#include <cstdio>
#include <vector>

using namespace lfgpu;

namespace {

template <bool MIXED, typename Limbs>
void add_cta(int threads, Limbs&& limbs, unsigned long long (&words)[2], bool& overflow) {
    constexpr int L = kLimbs<MIXED>;
    long long sum[L] = {};
    bool bad = false;
    for (int t = 0; t < threads; ++t) {
        int l[L];
        bad = !limbs(t, l) || bad;
        for (int j = 0; j < L; ++j) sum[j] += l[j];
    }
    int s[L];
    for (int j = 0; j < L; ++j) {
        s[j] = static_cast<int>(static_cast<unsigned>(sum[j]));  // what 32-bit additions leave
        overflow = overflow || (!bad && s[j] != sum[j]);
    }
    for (int w = 0; w < 2; ++w) words[w] += sum_word<MIXED>(s, w == 1, bad);
}

}  // namespace

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    FILE* in = std::fopen(argv[1], "rb");
    FILE* out = std::fopen(argv[2], "wb");
    if (!in || !out) return 2;
    long long cases = 0;
    if (std::fread(&cases, 8, 1, in) != 1) return 2;
    for (long long c = 0; c < cases; ++c) {
        long long head[3];
        double previous;
        if (std::fread(head, 8, 3, in) != 3 || std::fread(&previous, 8, 1, in) != 1) return 2;
        const int ctas = static_cast<int>(head[1]), threads = static_cast<int>(head[2]);
        std::vector<double> shares(static_cast<size_t>(ctas) * threads);
        if (std::fread(shares.data(), 8, shares.size(), in) != shares.size()) return 2;
        unsigned long long words[2] = {0, 0};
        bool overflow = false, ok;
        double total[2] = {0.0, 0.0};
        if (head[0]) {
            const float* pairs = reinterpret_cast<const float*>(shares.data());
            const int e = exponent_of_pair(static_cast<float>(previous));
            float up, down[2], hi, lo;
            pair_scale(e, up, down);
            for (int k = 0; k < ctas; ++k)
                add_cta<true>(
                    threads,
                    [&](int t, int(&l)[3]) {
                        const float* p = pairs + 2 * (static_cast<size_t>(k) * threads + t);
                        return pair_limbs(up, p[0], p[1], l);
                    },
                    words, overflow);
            ok = pair_total(down, words[0], words[1], ctas, hi, lo);
            total[0] = hi;
            total[1] = lo;
        } else {
            const int e = exponent_of(previous);
            for (int k = 0; k < ctas; ++k)
                add_cta<false>(
                    threads,
                    [&](int t, int(&l)[4]) { return fp64_limbs(e, shares[static_cast<size_t>(k) * threads + t], l); },
                    words, overflow);
            ok = fp64_total(e, words[0], words[1], ctas, total[0]);
        }
        ok = ok && ((words[0] >> 48) & 0xff) == 0 && ((words[1] >> 48) & 0xff) == 0 &&
             (words[0] >> 56) == static_cast<unsigned>(ctas);
        const double result[4] = {ok ? 1.0 : 0.0, overflow ? 1.0 : 0.0, total[0], total[1]};
        std::fwrite(result, 8, 4, out);
    }
    std::fclose(in);
    std::fclose(out);
    return 0;
}
