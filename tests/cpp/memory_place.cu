// Which caller memory the kernels read or write themselves, from what CUDA says
// about it, on the host.
#include <cstdio>

#include "gpma_internal.cuh"

int main() {
    struct Case {
        cudaMemoryType type;
        int device;
        bool read, written;  // by kernels on device 1
    };
    const Case cases[] = {
        {cudaMemoryTypeDevice, 1, true, true},        {cudaMemoryTypeDevice, 0, false, false},
        {cudaMemoryTypeDevice, 2, false, false},      {cudaMemoryTypeManaged, 1, true, false},
        {cudaMemoryTypeManaged, 0, true, false},      {cudaMemoryTypeHost, 1, false, false},
        {cudaMemoryTypeUnregistered, 1, false, false},
    };
    int bad = 0;
    for (const Case &c : cases) {
        cudaPointerAttributes a{};
        a.type = c.type;
        a.device = c.device;
        if (gpma::read_in_place(a, 1) != c.read || gpma::written_in_place(a, 1) != c.written) {
            std::printf("type %d on device %d\n", (int)c.type, c.device);
            bad = 1;
        }
    }
    if (!bad)
        std::puts("ok");
    return bad;
}
