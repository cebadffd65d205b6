// HostCopy (csrc/hostcopy.h) over tests/fake_cuda: argument is the copy's case.
// Prints "<bytes equal> <copies issued> <pending error after>".
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "hostcopy.h"

int main(int argc, char **argv)
{
    if(argc < 4) return 2;
    const size_t n = std::strtoull(argv[1], nullptr, 10);
    const int how = std::atoi(argv[2]);   // 0 pageable, 1 registered, 2 attributes fail, 3 no pinned memory
    const int before = std::atoi(argv[3]);
    std::vector<unsigned char> src(n), dst(n + 1, 7);
    for(size_t i = 0; i < n; ++i) src[i] = (unsigned char)(i * 2654435761u >> 13);
    fake::type = how == 1 ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    fake::no_attributes = how == 2;
    fake::no_host_alloc = how == 3;
    fake::pending = (cudaError_t)before;
    bhcb::HostCopy c;
    if(c.copy(dst.data(), src.data(), n, nullptr) != cudaSuccess) return 1;
    const cudaError_t after = fake::pending;
    std::printf("%d %d %d\n", std::memcmp(dst.data(), src.data(), n) == 0 && dst[n] == 7, fake::copies, (int)after);
    return 0;
}
