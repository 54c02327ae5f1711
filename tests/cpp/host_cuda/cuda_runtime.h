// The few names of the CUDA language that the headers under test need, for a
// host compiler: device code then is plain C++ run by host threads.
#pragma once

#define __host__
#define __device__
#define __shared__ static
#define __forceinline__ inline
#define __restrict__
#define __align__(n) alignas(n)

struct int2 {
    int x, y;
};
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
