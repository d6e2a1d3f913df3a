// Rys quadrature: roots and weights of the weight exp(-T t^2) on t in [0, 1]
// (Dupuis, Rys and King 1976): sum_r w_r x_r^m = F_m(T) for m < 2 NR, x = t^2.
//
// rys.cu tabulates x_r(T) and w_r(T) of every order as polynomials of degree
// RYS_DEG on intervals of width RYS_H (roots by the discretised Stieltjes
// procedure, Gautschi 1982, in long double; interpolation error below 2e-15
// relative).  From rys_tmax(NR) on the finite range no longer matters and the
// half-range Hermite limits x = X_r / T, w = W_r / sqrt(T) hold to 4e-15.
//
// Layout per order: X_r, W_r interleaved (2 NR doubles), then per interval
// RYS_DEG + 1 rows of 2 NR doubles (highest power first), so that the NR
// lanes of one quartet read one contiguous row per load.
#pragma once
#include "common.cuh"

namespace vlxb {

constexpr int RYS_MAX = 7;
constexpr int RYS_DEG = 9;
constexpr double RYS_H = 0.5;
constexpr double RYS_INV_H = 2.0;

__host__ __device__ constexpr double rys_tmax(int nr) { return 32.0 + 6.0 * nr; }
__host__ __device__ constexpr int rys_intervals(int nr) { return (int)(rys_tmax(nr) * RYS_INV_H); }
__host__ __device__ constexpr int rys_size(int nr) { return 2 * nr * (1 + rys_intervals(nr) * (RYS_DEG + 1)); }
__host__ __device__ constexpr int rys_offset(int nr)
{
    int o = 0;
    for (int n = 1; n < nr; n++) o += rys_size(n);
    return o;
}

// Device table of the current device (built and uploaded once), or null.
const double* rys_table_device();

// Root x = t^2 and weight of root r; tab is the table of order NR
// (rys_table_device() + rys_offset(NR)).
template <int NR>
__device__ __forceinline__ void rys_root(double T, const double* __restrict__ tab, int r, double& x, double& w)
{
    const double2* __restrict__ t2 = reinterpret_cast<const double2*>(tab);
    if (T < rys_tmax(NR)) {
        const int k = (int)(T * RYS_INV_H);
        const double s = fma(2.0 * RYS_INV_H, T, -(2.0 * k + 1.0));  // [-1, 1) on interval k
        const double2* row = t2 + NR + (k * (RYS_DEG + 1)) * NR + r;
        double2 c = __ldg(row);
        x = c.x;
        w = c.y;
#pragma unroll
        for (int j = 1; j <= RYS_DEG; j++) {
            c = __ldg(row + j * NR);
            x = fma(x, s, c.x);
            w = fma(w, s, c.y);
        }
    } else {
        const double2 c = __ldg(t2 + r);
        const double it = 1.0 / T;
        x = c.x * it;
        w = c.y * sqrt(it);
    }
}

// The same for an order known at run time; tab = rys_table_device().
__device__ __forceinline__ void rys_root_rt(int nr, double T, const double* __restrict__ tab, int r, double& x,
                                            double& w)
{
    switch (nr) {
        case 1: rys_root<1>(T, tab + rys_offset(1), r, x, w); break;
        case 2: rys_root<2>(T, tab + rys_offset(2), r, x, w); break;
        case 3: rys_root<3>(T, tab + rys_offset(3), r, x, w); break;
        case 4: rys_root<4>(T, tab + rys_offset(4), r, x, w); break;
        case 5: rys_root<5>(T, tab + rys_offset(5), r, x, w); break;
        case 6: rys_root<6>(T, tab + rys_offset(6), r, x, w); break;
        default: rys_root<7>(T, tab + rys_offset(7), r, x, w); break;
    }
}

}  // namespace vlxb
