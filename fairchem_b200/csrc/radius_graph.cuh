// Periodic-image arithmetic of the radius graph, shared by its kernels: which pairs are neighbours is decided by these
// expressions, each product and sum rounded separately.
#pragma once

#include "common.cuh"

namespace fcb200 {

struct Sys {
    int atom_begin, atom_end, r0, r1, r2, nimg, source_begin, grid_begin, d0, d1, d2;
    float ox, oy, oz, inv_h;
    float c[9];
};

__device__ __forceinline__ Sys load_sys(const int32_t* __restrict__ sys, int s) {
    const int32_t* w = sys + (int64_t)s * FCB200_SYS_WORDS;
    Sys v;
    v.atom_begin = w[0]; v.atom_end = w[1]; v.r0 = w[2]; v.r1 = w[3]; v.r2 = w[4]; v.nimg = w[5];
    v.source_begin = w[6]; v.grid_begin = w[7]; v.d0 = w[8]; v.d1 = w[9]; v.d2 = w[10];
    v.ox = __int_as_float(w[11]); v.oy = __int_as_float(w[12]); v.oz = __int_as_float(w[13]);
    v.inv_h = __int_as_float(w[14]);
#pragma unroll
    for (int i = 0; i < 9; ++i) v.c[i] = __int_as_float(w[15 + i]);
    return v;
}

__device__ __forceinline__ int find_system(const int32_t* __restrict__ sys, int nsys, int64_t sid) {
    int lo = 0, hi = nsys - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((int64_t)sys[(int64_t)mid * FCB200_SYS_WORDS + 6] <= sid) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ void decode_image(const Sys& s, int img, int& n0, int& n1, int& n2) {
    const int w2 = 2 * s.r2 + 1, w1 = 2 * s.r1 + 1;
    n2 = img % w2 - s.r2;
    img /= w2;
    n1 = img % w1 - s.r1;
    n0 = img / w1 - s.r0;
}

// position of periodic image (n0,n1,n2) of an atom; each product and sum rounded separately
__device__ __forceinline__ void image_position(const Sys& s, const float* __restrict__ pos, int atom, int n0, int n1, int n2,
                                               float& px, float& py, float& pz) {
    const float f0 = (float)n0, f1 = (float)n1, f2 = (float)n2;
    const float ox = __fadd_rn(__fadd_rn(__fmul_rn(f0, s.c[0]), __fmul_rn(f1, s.c[3])), __fmul_rn(f2, s.c[6]));
    const float oy = __fadd_rn(__fadd_rn(__fmul_rn(f0, s.c[1]), __fmul_rn(f1, s.c[4])), __fmul_rn(f2, s.c[7]));
    const float oz = __fadd_rn(__fadd_rn(__fmul_rn(f0, s.c[2]), __fmul_rn(f1, s.c[5])), __fmul_rn(f2, s.c[8]));
    px = __fadd_rn(pos[(int64_t)atom * 3 + 0], ox);
    py = __fadd_rn(pos[(int64_t)atom * 3 + 1], oy);
    pz = __fadd_rn(pos[(int64_t)atom * 3 + 2], oz);
}

__device__ __forceinline__ void grid_coords(const Sys& s, float px, float py, float pz, int& gx, int& gy, int& gz) {
    gx = (int)floorf((px - s.ox) * s.inv_h);
    gy = (int)floorf((py - s.oy) * s.inv_h);
    gz = (int)floorf((pz - s.oz) * s.inv_h);
}

__device__ __forceinline__ bool source_of(const int32_t* __restrict__ sys, int nsys, const float* __restrict__ pos, int64_t sid,
                                          Sys& s, float& px, float& py, float& pz, int& cell) {
    s = load_sys(sys, find_system(sys, nsys, sid));
    const int local = (int)(sid - s.source_begin);
    const int atom = s.atom_begin + local / s.nimg;
    int n0, n1, n2;
    decode_image(s, local % s.nimg, n0, n1, n2);
    image_position(s, pos, atom, n0, n1, n2, px, py, pz);
    int gx, gy, gz;
    grid_coords(s, px, py, pz, gx, gy, gz);
    if (gx < 0 || gy < 0 || gz < 0 || gx >= s.d0 || gy >= s.d1 || gz >= s.d2) {
        cell = -1;
        return false;
    }
    cell = s.grid_begin + gx + s.d0 * (gy + s.d1 * gz);
    return true;
}

__device__ __forceinline__ float dist_sq(float tx, float ty, float tz, float4 sp) {
    const float dx = __fsub_rn(tx, sp.x), dy = __fsub_rn(ty, sp.y), dz = __fsub_rn(tz, sp.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

}  // namespace fcb200
