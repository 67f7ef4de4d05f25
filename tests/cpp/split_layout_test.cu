// Host-side check of the split form's layout (jet_gb300/csrc/contract.cu): the
// word coordinates of its TMA boxes stay below 2^31 for every k, ranges of a
// cut k included, and paired planes are taken up to their limit.
#include "../../jet_gb300/csrc/contract.cu"

#include <cstdio>

using namespace jetgpu;

int main()
{
    const int precisions[] = {JETGPU_PREC_TF32X3, JETGPU_PREC_BF16X3, JETGPU_PREC_FP16X3};
    const int64_t quarter = 1ll << 29, half = 1ll << 30;
    const uint64_t ks[] = {32,
                           1024,
                           (uint64_t)quarter,
                           (uint64_t)(half - 65536),
                           (uint64_t)(half - 8192),
                           (uint64_t)(half - 32),
                           (uint64_t)half,
                           (uint64_t)(half + 32),
                           (uint64_t)(3 * quarter),
                           (uint64_t)(2 * half - 32)};
    int bad = 0, paired = 0;
    for (int prec : precisions)
        for (uint64_t k : ks) {
            const SplitLayout l = LayoutFor(prec, k, 4.0 * (double)k, 0);
            const uint64_t block = SplitPairWords(l.fmt), words = l.paired ? 2 : 1;
            const uint64_t stages = (k + block - 1) / block;
            // Ranges of a cut k: 1 (uncut) to one per SM of a whole GB300 (160).
            // An uncut k of any length is planar past the paired limit.
            for (uint64_t ranges : {1ull, 2ull, 132ull, 152ull, 160ull}) {
                if (ranges > 1 && !l.paired && k > 2 * (uint64_t)half - 16384)
                    continue; // TcSplits leaves it whole
                const uint64_t per = (stages + ranges - 1) / ranges;
                const uint64_t last = (per * ranges - 1) * block * words;
                if (last >= (1ull << 31)) {
                    std::printf("k %llu precision %d ranges %llu: coordinate %llu\n",
                                (unsigned long long)k, prec, (unsigned long long)ranges,
                                (unsigned long long)last);
                    ++bad;
                }
            }
            if (k <= (uint64_t)(half - 8192) && !l.paired) {
                std::printf("k %llu precision %d: not paired\n", (unsigned long long)k, prec);
                ++bad;
            }
            paired += l.paired;
            // 3M and the other main loops have no paired form.
            if (LayoutFor(prec, k, 1.0, 0, 0, JETGPU_ALGO_3M).paired ||
                LayoutFor(prec, k, 1.0, 1).paired)
                ++bad;
        }
    if (bad)
        return 1;
    std::printf("ok %d\n", paired);
    return 0;
}
