// Harness of block_select_reg (accel_common.cuh) for the tests: one selection
// per CTA over keys from global memory.
#include "accel_common.cuh"

namespace {

template <int NT, int NK>
__global__ void __launch_bounds__(NT) k_select(const uint32_t* keys, const int* n, const int* k, uint32_t* out) {
    __shared__ unsigned long long scratch[accel::kSelectScratch];
    // what an earlier kernel may have left there
    for (int i = threadIdx.x; i < accel::kSelectScratch; i += NT) scratch[i] = 0x5a5a5a5a5a5a5a5aull;
    __syncthreads();
    const int nb = n[blockIdx.x];
    const uint32_t* own = keys + (size_t)blockIdx.x * NT * NK;
    uint32_t key[NK];
    for (int j = 0; j < NK; j++) {
        const int i = (int)threadIdx.x + j * NT;
        key[j] = i < nb ? own[i] : 0xffffffffu;
    }
    const uint32_t v = accel::block_select_reg<NT, NK>(key, nb, k[blockIdx.x], scratch);
    out[(size_t)blockIdx.x * NT + threadIdx.x] = v;  // every thread has the result
}

}  // namespace

extern "C" int select_run(int nt, const uint32_t* keys, const int* n, const int* k, uint32_t* out, int blocks) {
    switch (nt) {
        case 32: k_select<32, 16><<<blocks, 32>>>(keys, n, k, out); break;
        case 64: k_select<64, 16><<<blocks, 64>>>(keys, n, k, out); break;
        case 256: k_select<256, 16><<<blocks, 256>>>(keys, n, k, out); break;
        case 512: k_select<512, 16><<<blocks, 512>>>(keys, n, k, out); break;
        default: return -1;
    }
    return (int)cudaDeviceSynchronize();
}
