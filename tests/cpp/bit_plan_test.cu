// Host-side check of the bit-permutation plan (jet_gb300/csrc/permute.cu): the
// kernel's offsets -- tile bases, runs and lanes -- replayed on the CPU for
// random power-of-2 shapes of 2^16 to 2^36 elements (past 2^32 the bases have
// high words), both element sizes, and compared with the plain
// permutation of index bits (output axis j = input axis perm[j]).
#include "../../jet_gb300/csrc/permute.cu"

#include <algorithm>
#include <cstdio>
#include <random>

using namespace jetgpu;

int main()
{
    std::mt19937_64 rng(7);
    int plans = 0;
    for (int rep = 0; rep < 4000; ++rep) {
        const int n = 16 + (int)(rng() % 21);
        std::vector<uint64_t> shape;
        std::vector<int> logd;
        for (int left = n; left > 0;) {
            const int d = 1 + (int)(rng() % std::min(left, 1 + (int)(rng() % 6)));
            shape.push_back(1ull << d);
            logd.push_back(d);
            left -= d;
        }
        const int r = (int)shape.size();
        std::vector<int32_t> perm(r);
        for (int i = 0; i < r; ++i)
            perm[i] = i;
        if (rep % 3) // else rotations of long runs
            std::shuffle(perm.begin(), perm.end(), rng);
        else
            std::rotate(perm.begin(), perm.begin() + rng() % r, perm.end());
        const int log_ve = rep & 1;
        Simplified s;
        static BitParams p;
        if (Simplify(r, shape.data(), perm.data(), s) != JETGPU_OK)
            return 1;
        if (!BuildBitParams(s, 1, log_ve, p)) {
            if (n >= 17 + log_ve && n <= 35) {
                std::printf("no plan for 2^%d\n", n);
                return 1;
            }
            continue;
        }
        ++plans;
        if (p.n != n || p.n_seg > kMaxOuter || p.total_tiles != 1ull << (n - p.u)) {
            std::printf("bad plan\n");
            return 1;
        }
        // Bit of the input index that output bit o holds.
        std::vector<int> in_off(r), src(n);
        for (int i = r - 1, o = 0; i >= 0; --i) {
            in_off[i] = o;
            o += logd[i];
        }
        for (int j = r - 1, o = 0; j >= 0; --j)
            for (int q = 0; q < logd[perm[j]]; ++q)
                src[o++] = in_off[perm[j]] + q;
        for (int k = 0; k < 64; ++k) {
            const uint32_t tt = (uint32_t)(rng() % p.total_tiles);
            uint64_t bi = 0, bo = 0;
            for (int lane = 0; lane < 32; ++lane) {
                const BitSegment seg(p, lane);
                bi |= seg.In(tt);
                bo |= seg.Out(tt);
            }
            if (n <= 32 && ((bi | bo) >> 32)) {
                std::printf("2^%d: an offset past 32 bits\n", n);
                return 1;
            }
            const int h = (int)(rng() % (1u << (p.u - p.t)));
            const uint32_t m = (uint32_t)(rng() % (1u << p.t));
            uint32_t L = p.l_hi[h];
            for (int j = 0; j < p.t; ++j)
                L |= ((m >> j) & 1u) << p.lo_pos[j];
            const uint64_t out = bo + p.out_hi[h] + m;
            const uint64_t in = bi + p.in_hi[L >> p.t] + (L & ((1u << p.t) - 1));
            uint64_t want = 0;
            for (int o = 0; o < n; ++o)
                want |= ((out >> o) & 1ull) << src[o];
            if (out >> n || in != want || L >= 1u << p.u) {
                std::printf("2^%d tile %u run %d lane %u: %llu, want %llu\n", n, tt, h, m,
                            (unsigned long long)in, (unsigned long long)want);
                return 1;
            }
        }
    }
    std::printf("ok %d plans\n", plans);
    return plans > 3000 ? 0 : 1;
}
