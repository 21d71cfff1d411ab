// Two groups of 128 threads behind two other warps, as the product's epilogue, vote several times over their own barriers:
// thread t of a group says yes in round r where bit t of yes[r * 2 + group] is set.  Every thread's answer goes to `out`.
#include "../../cnet_b200/csrc/common.cuh"

__global__ void vote_k(const uint4* yes, int rounds, unsigned char* out) {
    if (threadIdx.x < 64) return;
    const int e = threadIdx.x - 64, group = e >> 7, t = e & 127;
    for (int r = 0; r < rounds; ++r) {
        const uint4 y = yes[2 * r + group];
        const unsigned word = t < 32 ? y.x : t < 64 ? y.y : t < 96 ? y.z : y.w;
        out[(2 * r + group) * 128 + t] = cnb_group_any(1 + group, 128, word >> (t & 31) & 1) ? 1 : 0;
    }
}

extern "C" int vote(const void* yes, int rounds, void* out, void* stream) {
    vote_k<<<1, 64 + 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(static_cast<const uint4*>(yes), rounds, static_cast<unsigned char*>(out));
    return (int) cudaGetLastError();
}
