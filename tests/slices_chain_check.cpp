/* Host check of sliced plans whose rows differ in length: every nonzero in
 * exactly one lane, every row finished once, and no lane with more than `chain`
 * entries unless its row already has all 32 lanes. */
#include "../pdal_gb300/csrc/common.h"
#include "../pdal_gb300/csrc/rowblock_config.h"

#include <random>

using namespace pdal;
#define CHECK(c)                                                    \
    do {                                                            \
        if (!(c)) {                                                 \
            std::printf("line %d, trial %d: %s\n", __LINE__, trial, #c); \
            return 1;                                               \
        }                                                           \
    } while (0)

int main() {
    std::mt19937 gen(2);
    for (int trial = 0; trial < 300; ++trial) {
        /* rows of 0 to 20 entries and, one in 2 to 200, of up to S + 100 */
        const int nr = 1 + gen() % 4000, S = 256 << (gen() % 4), every = 2 + gen() % 200;
        std::vector<int> rp(nr + 1, 0);
        for (int i = 0; i < nr; ++i) rp[i + 1] = rp[i] + (int)(gen() % every == 0 ? gen() % (S + 100) : gen() % 21);
        const int lanes = 1 << (gen() % 6), chain = 8 << (gen() % 3);
        const HostPlan P = plan_rows(nr, rp.data(), S);
        const HostSlices Q = plan_slices(P, rp.data(), lanes, chain);
        std::vector<int> seen(rp[nr], 0), rows(nr, 0);
        long long len = 0;
        for (int s = 0; s < Q.n; ++s) {
            const int *d = &Q.desc[4 * (size_t)s];
            CHECK(d[0] == len);
            len += 32LL * d[1];
            int most = 0;
            for (int l = 0; l < 32; ++l) {
                const int r = Q.rl[64 * (size_t)s + 2 * l], c = Q.rl[64 * (size_t)s + 2 * l + 1];
                CHECK(c >= 0 && c <= d[1]);
                most = std::max(most, c);
                if (d[2] == 0) { /* a part of a long row */
                    const int *li = &P.linfo[4 * (size_t)r];
                    rows[li[0]] += l == 0 && d[3] == 8 * li[2];
                    for (int j = 0; j < c; ++j) seen[li[3] + (d[3] / 8 - li[2]) * S + (d[3] & 7) * 32 + l + j * kThreads]++;
                    continue;
                }
                CHECK(d[2] >= lanes && d[2] <= 32);
                if (r < 0) {
                    CHECK(c == 0);
                    continue;
                }
                CHECK(c <= chain || d[2] == 32);
                CHECK(d[2] == lanes || rp[r + 1] - rp[r] > d[2] / 2 * chain);
                rows[r] += (l & (d[2] - 1)) == 0;
                for (int j = 0; j < c; ++j) seen[rp[r] + (l & (d[2] - 1)) + j * d[2]]++;
            }
            CHECK(d[2] == 0 || most == d[1]); /* no padding but that of the shorter lanes */
        }
        CHECK(len == Q.len);
        for (int v : seen) CHECK(v == 1);
        for (int v : rows) CHECK(v == 1);
    }
    std::puts("ok");
    return 0;
}
