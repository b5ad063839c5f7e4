// bmxg_fx.cuh -- the list path's 64-bit fixed-point positions back to FP64
// (FxGeom), shared by the list kernels and the store of the state.
#pragma once
#include "bmxg_kernels.cuh"

namespace bmxg {

__device__ __forceinline__ unsigned long long fx_join(unsigned h, unsigned l)
{
    return ((unsigned long long)h << 32) | l;
}

// x of a fixed-point coordinate: o + X span / 2^64, the product X ms 2^(es - 64)
// rounded to nearest even once (then the FP64 addition of a non-zero origin);
// a periodic coordinate is kept below phi.
__device__ __forceinline__ double from_fx(unsigned long long X, const FxGeom &F, int ax)
{
    const unsigned long long ms = F.ms[ax];
    const unsigned long long hi = __umul64hi(X, ms), lo = X * ms;
    unsigned long long t, rest;
    int E;  // value = t 2^E with t in [2^63, 2^64), rest the bits below t
    if (hi) {
        const int lz = __clzll((long long)hi);
        t = lz ? ((hi << lz) | (lo >> (64 - lz))) : hi;
        rest = lo << lz;
        E = F.es[ax] - lz;
    } else if (lo) {
        const int lz = __clzll((long long)lo);
        t = lo << lz;
        rest = 0ull;
        E = F.es[ax] - 64 - lz;
    } else {
        t = 0ull;
        rest = 0ull;
        E = 0;
    }
    double v = 0.0;
    if (t) {
        unsigned long long m = t >> 11;
        const unsigned long long rb = (t >> 10) & 1ull;
        const bool sticky = (t & 0x3ffull) != 0ull || rest != 0ull;
        m += rb & ((sticky ? 1ull : 0ull) | (m & 1ull));
        if (m >> 53) {
            m >>= 1;
            ++E;
        }
        v = __longlong_as_double((long long)((((unsigned long long)(E + 1086)) << 52) | (m & 0xfffffffffffffull)));
    }
    if (F.ozero[ax]) {
        // (periodic with plo = 0: v < len unless rounding reached it)
        if (F.per[ax] && !(v < F.phi[ax])) v = nextafter(F.phi[ax], 0.0);
        return v;
    }
    double x = F.o[ax] + v;
    if (F.per[ax] && !(x < F.phi[ax])) x = nextafter(F.phi[ax], -1.0e300);
    return x;
}

}  // namespace bmxg
