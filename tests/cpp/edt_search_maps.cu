// The distance transform's searches (edt_search_check.cu's check) on whole maps: those given, and maps of up to
// 4096 x 4096 whose distances reach their diagonals or whose rows meet hardly any occupied column.
//
//   edt_search_maps [occupancy.u8 W H]...      (x-major, 1 = occupied)
#define main edt_search_check_main
#include "edt_search_check.cu"
#undef main

#include <cstdlib>

int main(int argc, char** argv) {
    for (int a = 1; a + 2 < argc; a += 3) {
        const int W = atoi(argv[a + 1]), H = atoi(argv[a + 2]);
        std::vector<uint8_t> occ((size_t)W * H);
        FILE* f = fopen(argv[a], "rb");
        if (!f || fread(occ.data(), 1, occ.size(), f) != occ.size()) {
            printf("cannot read %s\n", argv[a]);
            return 2;
        }
        fclose(f);
        check(occ, W, H, argv[a]);
    }
    std::mt19937_64 rng(12345);
    const int dims[][2] = {{2048, 2048}, {4096, 4096}, {1001, 4096}, {5000, 1500}};
    for (auto& dd : dims)
        for (int pat = 0; pat < 3; ++pat) {
            const int W = dd[0], H = dd[1];
            if (W == 4096 && pat == 1) continue;
            std::vector<uint8_t> occ((size_t)W * H, 0);
            if (pat == 0) occ[0] = 1;   // a corner: distances up to the diagonal
            if (pat == 1)               // three columns with five cells each
                for (int c = 0; c < 3; ++c) {
                    const int x = (int)(rng() % W);
                    for (int i = 0; i < 5; ++i) occ[(size_t)x * H + rng() % H] = 1;
                }
            if (pat == 2) {             // the last cell, and a row met here and there
                occ[(size_t)(W - 1) * H + H - 1] = 1;
                const int y = (int)(rng() % H);
                for (int x = 0; x < W; x += 1 + (int)(rng() % 700)) occ[(size_t)x * H + y] = 1;
            }
            check(occ, W, H, "whole");
        }
    printf("%d cases, %d mismatches\n", cases, fails);
    return fails != 0;
}
