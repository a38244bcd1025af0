// Host check of the distance transform's searches (rlc_map.cu: edt_col_search, edt_row_search, as
// k_edt_cols and k_edt_rows call them for maps up to 16384 per side) against the oracle's
// Felzenszwalb-Huttenlocher transform, bit for bit.  Every map runs with the form launch_edt picks
// for its sides and, where that is the exact one, with rounded keys too.
//
// Prints "<cases> cases, <n> mismatches" and exits non-zero on a mismatch.
#include "rlc_map.cu"

#include <cmath>
#include <cstring>
#include <random>
#include <vector>

extern "C" void orc_edt(const uint8_t* occ, int width, int height, float* dt_out);

namespace rlc {
int set_last_error(int code, const char*) { return code; }   // the map entry points are not called here
}

namespace {

int cases = 0, fails = 0;

void check(const std::vector<uint8_t>& occ, int W, int H, const char* what) {
    std::vector<float> ref((size_t)W * H);
    orc_edt(occ.data(), W, H, ref.data());
    const int nb = (W + rlc::kEdtBlock - 1) / rlc::kEdtBlock, nf = (W + rlc::kEdtFar - 1) / rlc::kEdtFar;
    std::vector<uint16_t> g((size_t)W * H), gmin((size_t)nb * H, 0xFFFF), gfar((size_t)nf * H, 0xFFFF);
    for (int x = 0; x < W; ++x) {
        const uint8_t* col = occ.data() + (size_t)x * H;
        std::vector<int> prev(H);
        std::vector<unsigned> next(H);
        int p = -1;
        for (int q = 0; q < H; ++q) { if (col[q]) p = q; prev[q] = p; }
        unsigned n = rlc::kEdtNone;
        for (int q = H - 1; q >= 0; --q) { if (col[q]) n = (unsigned)q; next[q] = n; }
        for (int q = 0; q < H; ++q) {
            g[(size_t)x * H + q] = (uint16_t)rlc::edt_col_search(prev[q], next[q], q, H, [&](int r) { return col[r] != 0; });
            uint16_t& m = gmin[(size_t)(x / rlc::kEdtBlock) * H + q];
            m = std::min(m, g[(size_t)x * H + q]);
            uint16_t& f = gfar[(size_t)(x / rlc::kEdtFar) * H + q];
            f = std::min(f, g[(size_t)x * H + q]);
        }
    }
    const bool exact = (long long)(W - 1) * (W - 1) + (long long)(H - 1) * (H - 1) < (1ll << 24);
    const int slack = W <= rlc::kEdtExactSide && H <= rlc::kEdtExactSide ? 1 : 24;
    for (int form = exact ? 0 : 1; form < 2; ++form) {
        size_t bad = 0;
        for (int y = 0; y < H; ++y) {
            const auto gy = [&](int q) { return (unsigned)g[(size_t)q * H + y]; };
            const auto my = [&](int b) { return (unsigned)gmin[(size_t)b * H + y]; };
            const auto fy = [&](int b) { return (unsigned)gfar[(size_t)b * H + y]; };
            for (int x = 0; x < W; ++x) {
                const float v = sqrtf(form == 0 ? rlc::edt_row_search<true>(gy, my, fy, W, x, 0)
                                                : rlc::edt_row_search<false>(gy, my, fy, W, x, slack));
                const float* r = &ref[(size_t)x * H + y];
                if (memcmp(&v, r, sizeof(float)) != 0 && bad++ == 0)
                    printf("mismatch %s %dx%d form %d at (%d, %d): %.9g vs %.9g\n", what, W, H, form, x, y, v, *r);
            }
        }
        ++cases;
        fails += bad != 0;
    }
}

}  // namespace

int main() {
    std::mt19937_64 rng(4711);
    const int sizes[][2] = {{1, 1}, {1, 9}, {9, 1}, {2, 2}, {31, 33}, {32, 8}, {33, 31}, {64, 65}, {65, 64}, {97, 130}, {300, 200}};
    const double dens[] = {0.0, 1.0, 0.0005, 0.01, 0.2, 0.9};
    for (auto& s : sizes)
        for (double d : dens) {
            std::vector<uint8_t> occ((size_t)s[0] * s[1]);
            std::bernoulli_distribution b(d);
            for (auto& o : occ) o = b(rng);
            check(occ, s[0], s[1], "random");
        }
    for (int t = 0; t < 60; ++t) {   // a few obstacles far apart, sometimes a full column: blocks are opened
        const int W = 1 + (int)(rng() % 700), H = 1 + (int)(rng() % 120);
        std::vector<uint8_t> occ((size_t)W * H, 0);
        for (int i = (int)(rng() % 5); i > 0; --i) occ[(rng() % W) * (size_t)H + rng() % H] = 1;
        if (t % 6 == 0) {
            const size_t x = rng() % W;
            for (int y = 0; y < H; ++y) occ[x * H + y] = 1;
        }
        check(occ, W, H, "sparse");
    }
    // keys that round: sides at and above the exact limits, obstacles that put distances and squares
    // near 2^24 .. 2^28
    const int dims[][2] = {{4096, 24}, {24, 4096}, {4097, 24}, {24, 4097}, {4096, 300}, {10976, 20}, {20, 10976}, {16384, 9}, {9, 16384}, {6000, 700}};
    for (auto& dd : dims)
        for (int pat = 0; pat < 4; ++pat) {
            const int W = dd[0], H = dd[1];
            if ((size_t)W * H > 1000000 && pat > 1) continue;
            std::vector<uint8_t> occ((size_t)W * H, 0);
            if (pat == 0)
                for (int i = 0; i < 6; ++i) occ[(rng() % W) * (size_t)H + rng() % H] = 1;
            if (pat == 1) {
                std::bernoulli_distribution b(0.004);
                for (auto& o : occ) o = b(rng);
            }
            if (pat == 2) occ[0] = 1;
            if (pat == 3)
                for (int i = 0; i < 40; ++i) {   // pairs of obstacles, each way from some cell almost equally far
                    occ[(rng() % W) * (size_t)H + H - 1] = 1;
                    occ[(size_t)(W - 1) * H + rng() % H] = 1;
                }
            check(occ, W, H, "large");
        }
    printf("%d cases, %d mismatches\n", cases, fails);
    return fails != 0;
}
