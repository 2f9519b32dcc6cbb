// The block kernel's first items: every item below the grid's size is exactly one
// block's, and packed, the blocks b and b + (grid + 1) / 2 have neighbours.  Host code only.
#include "kernels.cuh"

#include <cstdio>
#include <vector>

int main()
{
    for (int grid = 1; grid <= 700; ++grid)
        for (int packed = 0; packed < 2; ++packed) {
            std::vector<int> seen((size_t)grid, 0);
            for (int b = 0; b < grid; ++b) {
                const int q = ga::first_item(b, grid, packed != 0);
                if (q < 0 || q >= grid || seen[(size_t)q]++) return 1;
                const int second = b + (grid + 1) / 2;
                if (packed && second < grid && ga::first_item(second, grid, true) != q + 1) return 2;
            }
        }
    std::puts("ok");
    return 0;
}
