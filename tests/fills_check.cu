// The words a batch's first kernel sets: as many as Fills holds are launched, one more
// is refused before any launch.  Host code only, linked with fake_cudart.cpp.
#include "kernels.cuh"

#include <cstdio>

int main()
{
    ga::PairDesc D{};
    D.n = 1;
    int32_t words[ga::Fills::MAX + 1];
    ga::Fills F;
    for (int k = 0; k < ga::Fills::MAX; ++k) F.add(words + k, 1, k);
    if (ga::launch_pack(D, 64, nullptr, nullptr, nullptr, F) != cudaSuccess) return 1;
    F.add(words + ga::Fills::MAX, 1, 0);
    if (F.count != ga::Fills::MAX) return 2;
    if (ga::launch_pack(D, 64, nullptr, nullptr, nullptr, F) == cudaSuccess) return 3;
    std::puts("ok");
    return 0;
}
