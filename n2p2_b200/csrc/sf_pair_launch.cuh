// Launcher of one instantiation of the two-pass symmetry-function kernels
// (M1, M4: blocks per SM that the kernels with one and with four warps per atom
// are compiled for).
#pragma once

#include <algorithm>

#include "sf_pair.cuh"

static_assert(sizeof(n2p2b::sfp2::Head) * n2p2b::sfp2::kW + 64 <= 1024,
              "static shared memory beyond what kPairSmemBlock leaves");

#define N2P2B_PAIR_LAUNCH(NAME, R, CT, NZ, KINDS, M1, M4)                     \
    void pairLaunch_##NAME(int pass, SFParams const& P, PairParams const& T,  \
                           PairLaunch const& L, int shm, cudaStream_t s)      \
    {                                                                         \
        auto k = pass == 0                                                    \
            ? (L.wpa == 1 ? sfp2::pairValueKernel<R, CT, NZ, KINDS, 1, M1>    \
                          : sfp2::pairValueKernel<R, CT, NZ, KINDS, 4, M4>)   \
            : (L.wpa == 1 ? sfp2::pairTermKernel<R, CT, NZ, KINDS, 1, M1>     \
                          : sfp2::pairTermKernel<R, CT, NZ, KINDS, 4, M4>);   \
        /* One value for all callers: threads share the kernel's attribute. */ \
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                             kPairSmemBlock);                                 \
        int per = 0;                                                          \
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, sfp2::kT, shm); \
        int const atoms = 4 / L.wpa;                                          \
        int const grid = std::min((L.n + atoms - 1) / atoms,                  \
                                  std::max(1, per) * L.sms);                  \
        k<<<grid, sfp2::kT, shm, s>>>(P, T, L);                               \
    }
