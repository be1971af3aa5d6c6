/* Host check of the sliced plans: every nonzero in exactly one lane, every
 * row finished exactly once, packed positions dense, CTA ranges in order. */
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
    std::mt19937 gen(1);
    for (int trial = 0; trial < 400; ++trial) {
        /* short rows, few long ones, middling ones, only empty ones */
        const int nr = 1 + gen() % 3000, S = 256 << (gen() % 4), mode = gen() % 4;
        std::vector<int> rp(nr + 1, 0);
        for (int i = 0; i < nr; ++i) {
            const int len = mode == 0   ? gen() % 20
                            : mode == 1 ? (gen() % 50 == 0 ? gen() % 9000 : gen() % 3)
                            : mode == 2 ? gen() % 600
                                        : 0;
            rp[i + 1] = rp[i] + len;
        }
        const int lanes = trial % 3 == 0 ? 0 : 1 << (gen() % 6);
        const HostPlan P = plan_rows(nr, rp.data(), S);
        const HostSlices Q = plan_slices(P, rp.data(), lanes);
        std::vector<int> seen(rp[nr], 0), rows(nr, 0);
        long long len = 0;
        for (int s = 0; s < Q.n; ++s) {
            const int *d = &Q.desc[4 * (size_t)s];
            CHECK(d[0] == len);
            len += 32LL * d[1];
            for (int l = 0; l < 32; ++l) {
                const int r = Q.rl[64 * (size_t)s + 2 * l], c = Q.rl[64 * (size_t)s + 2 * l + 1];
                CHECK(c >= 0 && c <= d[1]);
                int k, step, end;
                if (d[2] > 0) {
                    if (r < 0) {
                        CHECK(c == 0);
                        continue;
                    }
                    CHECK(r < nr && (lanes == 0 || d[2] == lanes));
                    rows[r] += (l & (d[2] - 1)) == 0;
                    k = rp[r] + (l & (d[2] - 1));
                    step = d[2];
                    end = rp[r + 1];
                } else {
                    const int *li = &P.linfo[4 * (size_t)r];
                    CHECK(d[3] / 8 < P.npieces);
                    rows[li[0]] += l == 0 && d[3] == 8 * li[2];
                    k = li[3] + (d[3] / 8 - li[2]) * S + (d[3] & 7) * 32 + l;
                    step = kThreads;
                    end = rp[li[0] + 1];
                }
                for (int j = 0; j < c; ++j) {
                    CHECK(k + j * step < end);
                    seen[k + j * step]++;
                }
            }
        }
        CHECK(len == Q.len);
        for (int v : seen) CHECK(v == 1);
        for (int v : rows) CHECK(v == 1);
        for (int parts : {1, 3, 152}) {
            long long most = 0;
            const std::vector<int> cut = split_slices(Q, parts, most);
            CHECK(cut[0] == 0 && cut[parts] == Q.n);
            for (int p = 0; p < parts; ++p) CHECK(cut[p] <= cut[p + 1]);
        }
    }
    std::puts("ok");
    return 0;
}
