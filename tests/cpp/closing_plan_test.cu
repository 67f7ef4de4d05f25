// Host-side check of closing_kernel's plan (jet_gb300/csrc/gemm_simt.cu): every
// element that its copies read, replayed on the CPU for random power-of-2
// shapes and axis orders, both element sizes, against the permuted operands'
// own indices -- A and B of a tile's row are the same k, every k comes once,
// rows and columns are where the product looks, and no two elements share a
// place in shared memory. Forms that the plan must refuse are refused.
#include "../../jet_gb300/csrc/gemm_simt.cu"

#include <cstdio>
#include <random>
#include <set>

using namespace jetgpu;

// A random shape of 2^total elements whose first (lead) or last axes in
// permuted order make 2^split.
static void RandomOperand(std::mt19937_64 &rng, int lead, int tail, std::vector<uint64_t> &shape,
                          std::vector<int32_t> &perm)
{
    std::vector<uint64_t> permuted;
    for (int part : {lead, tail})
        for (int left = part; left > 0;) {
            const int d = 1 + (int)(rng() % std::min(left, 3));
            permuted.push_back(1ull << d);
            left -= d;
        }
    if (rng() % 4 == 0)
        permuted.push_back(1);
    const int r = (int)permuted.size();
    perm.resize(r);
    shape.resize(r);
    for (int i = 0; i < r; ++i)
        perm[i] = i;
    std::shuffle(perm.begin(), perm.end(), rng);
    for (int j = 0; j < r; ++j)
        shape[perm[j]] = permuted[j];
}

// Permuted index of every element of memory.
static std::vector<uint32_t> PermutedIndex(const std::vector<uint64_t> &shape,
                                           const std::vector<int32_t> &perm)
{
    const int r = (int)shape.size();
    uint64_t total = 1;
    for (uint64_t d : shape)
        total *= d;
    std::vector<uint32_t> out(total);
    std::vector<uint64_t> digit(r);
    for (uint64_t off = 0; off < total; ++off) {
        uint64_t left = off;
        for (int i = r - 1; i >= 0; --i) {
            digit[i] = left % shape[i];
            left /= shape[i];
        }
        uint64_t at = 0;
        for (int j = 0; j < r; ++j)
            at = at * shape[perm[j]] + digit[perm[j]];
        out[off] = (uint32_t)at;
    }
    return out;
}

template <typename V>
static bool Replay(const ClosingPlan &p, const std::vector<uint32_t> &ai,
                   const std::vector<uint32_t> &bi, int m, int n, int k, int klog, int mt, int nt)
{
    const int KC = 1 << klog, tiles = k >> klog;
    std::vector<char> seen(k, 0);
    uint32_t a_base = 0, b_base = 0;
    for (int t = 0; t < tiles; ++t) {
        uint32_t fa = 0, fb = 0; // the start of a range
        for (int b = 0; b < p.tile_bits; ++b)
            if (t >> b & 1) {
                fa += p.a.tile[b];
                fb += p.b.tile[b];
            }
        if (fa != a_base || fb != b_base)
            return false;
        std::vector<int> krow(KC, -1);
        std::set<int> places;
        for (int e = 0; e < m * KC; ++e) {
            uint32_t src, at;
            ClosingElement(p.a, e, 0, 11, src, at);
            const int dst = (int)at;
            const uint64_t off = (uint64_t)a_base + src;
            if (off >= ai.size() || !places.insert(dst).second)
                return false;
            const int i = (int)(ai[off] / k), kv = (int)(ai[off] % k);
            int kk = 0;
            while (kk + 1 < KC && ClosingRow<V>(kk + 1, mt) <= dst)
                ++kk;
            if (dst != ClosingRow<V>(kk, mt) + i || (krow[kk] >= 0 && krow[kk] != kv))
                return false;
            krow[kk] = kv;
        }
        places.clear();
        for (int e = 0; e < n * KC; ++e) {
            uint32_t src, at;
            ClosingElement(p.b, e, 0, 11, src, at);
            const int dst = (int)at;
            const uint64_t off = (uint64_t)b_base + src;
            if (off >= bi.size() || !places.insert(dst).second)
                return false;
            const int kv = (int)(bi[off] / n), j = (int)(bi[off] % n);
            int kk = 0;
            while (kk + 1 < KC && ClosingRow<V>(kk + 1, nt) <= dst)
                ++kk;
            if (dst != ClosingRow<V>(kk, nt) + j || krow[kk] != kv)
                return false;
        }
        for (int kk = 0; kk < KC; ++kk) {
            if (krow[kk] < 0 || seen[krow[kk]])
                return false;
            seen[krow[kk]] = 1;
        }
        int ones = 0;
        while (t >> ones & 1)
            ++ones;
        a_base += p.a.step[ones];
        b_base += p.b.step[ones];
    }
    return std::count(seen.begin(), seen.end(), 1) == k;
}

int main()
{
    std::mt19937_64 rng(11);
    int plans = 0;
    for (int rep = 0; rep < 240; ++rep) {
        const int nm = 1 + (int)(rng() % 5);
        const int nn = nm == 5 ? 1 + (int)(rng() % 4) : 1 + (int)(rng() % 5);
        const int nk = 11 + (int)(rng() % 3);
        std::vector<uint64_t> as, bs;
        std::vector<int32_t> ap, bp;
        RandomOperand(rng, nm, nk, as, ap);
        RandomOperand(rng, nk, nn, bs, bp);
        const int m = 1 << nm, n = 1 << nn, k = 1 << nk;
        int mt, nt;
        SmallTile(m, n, k, mt, nt);
        const auto ai = PermutedIndex(as, ap), bi = PermutedIndex(bs, bp);
        for (int klog : {kClosingLog<float>, kClosingLog<double>}) {
            ClosingPlan p;
            if (!PlanClosing((int)as.size(), as.data(), ap.data(), (int)bs.size(), bs.data(),
                             bp.data(), m, n, k, klog, p)) {
                printf("refused m %d n %d k %d\n", m, n, k);
                return 1;
            }
            const bool ok = klog == kClosingLog<float>
                                ? Replay<float2>(p, ai, bi, m, n, k, klog, mt, nt)
                                : Replay<double2>(p, ai, bi, m, n, k, klog, mt, nt);
            if (!ok) {
                printf("wrong element: rep %d m %d n %d k %d klog %d\n", rep, m, n, k, klog);
                return 1;
            }
            ++plans;
        }
    }
    // The largest operands: bases within 2^31, steps back to the sum of bits.
    {
        const std::vector<uint64_t> as = {1ull << 26, 32}, bs = {16, 1ull << 26};
        const int32_t ap[] = {1, 0}, bp[] = {1, 0};
        ClosingPlan p;
        if (!PlanClosing(2, as.data(), ap, 2, bs.data(), bp, 32, 16, 1ull << 26, 6, p))
            return 2;
        uint32_t base = 0;
        for (uint32_t t = 0; t + 1 < (1u << p.tile_bits); ++t) {
            int ones = 0;
            while (t >> ones & 1)
                ++ones;
            base += p.a.step[ones];
        }
        uint32_t last = 0;
        for (int b = 0; b < p.tile_bits; ++b)
            last += p.a.tile[b];
        if (base != last || (uint64_t)last >= (32ull << 26))
            return 2;
    }
    // Refused: extents not powers of 2, short k, vectors, too large outputs or operands.
    const auto refused = [](std::vector<uint64_t> as, std::vector<uint64_t> bs, uint64_t m,
                            uint64_t n, uint64_t k) {
        const int32_t turn[] = {1, 0};
        ClosingPlan p;
        return !PlanClosing(2, as.data(), turn, 2, bs.data(), turn, m, n, k, 6, p);
    };
    if (!refused({2187, 4}, {4, 2187}, 4, 4, 2187) || !refused({4096, 3}, {4, 4096}, 3, 4, 4096) ||
        !refused({1024, 4}, {4, 1024}, 4, 4, 1024) || !refused({4096, 1}, {4, 4096}, 1, 4, 4096) ||
        !refused({4096, 4}, {1, 4096}, 4, 1, 4096) ||
        !refused({4096, 32}, {32, 4096}, 32, 32, 4096) ||
        !refused({1ull << 30, 4}, {4, 1ull << 30}, 4, 4, 1ull << 30))
        return 3;
    printf("ok %d plans\n", plans);
    return 0;
}
