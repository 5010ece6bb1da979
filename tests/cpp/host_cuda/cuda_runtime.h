// What pow_pos.cuh needs of CUDA, for compiling it as host code.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __forceinline__ inline

struct alignas(16) double2 {
    double x, y;
};
template <typename T>
inline T __ldg(const T* p) { return *p; }
inline uint64_t bits_of(double x) {
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
}
inline int __double2hiint(double x) { return static_cast<int>(bits_of(x) >> 32); }
inline int __double2loint(double x) { return static_cast<int>(bits_of(x)); }
inline double __hiloint2double(int hi, int lo) {
    const uint64_t u = static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32 | static_cast<uint32_t>(lo);
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}
