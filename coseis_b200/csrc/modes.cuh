// Corner modes of a cell (see modal.cuh): three-component values and the sums
// and differences that the modes are made of.
#pragma once

namespace sordgpu {

// A vector, operated on by component.
struct M3 {
    float x, y, z;
};
__device__ __forceinline__ M3 operator+(const M3& a, const M3& b) { return M3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ M3 operator-(const M3& a, const M3& b) { return M3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ M3 operator-(const M3& a) { return M3{-a.x, -a.y, -a.z}; }
__device__ __forceinline__ M3 operator*(float a, const M3& b) { return M3{a * b.x, a * b.y, a * b.z}; }
__device__ __forceinline__ M3 m_fma(float a, const M3& b, const M3& c) {
    return M3{fmaf(a, b.x, c.x), fmaf(a, b.y, c.y), fmaf(a, b.z, c.z)};
}

// In-plane sums of the four corner values (0,0) (1,0) (0,1) (1,1) of a node
// plane: (const, j, k, jk), or without the constant.
__device__ __forceinline__ void m_sums4(const M3 (&c)[4], M3 (&o)[4]) {
    const M3 d0 = c[1] - c[0], d1 = c[3] - c[2], s0 = c[0] + c[1], s1 = c[2] + c[3];
    o[0] = s0 + s1;
    o[1] = d0 + d1;
    o[2] = s1 - s0;
    o[3] = d1 - d0;
}
__device__ __forceinline__ void m_sums3(const M3 (&c)[4], M3 (&o)[3]) {
    const M3 d0 = c[1] - c[0], d1 = c[3] - c[2], s0 = c[0] + c[1], s1 = c[2] + c[3];
    o[0] = d0 + d1;
    o[1] = s1 - s0;
    o[2] = d1 - d0;
}

// Sums of one mode pair: p keeps its sign across the cell, q changes it.
// T completes the lower plane, acc starts the upper one.
template <bool P, bool Q>
__device__ __forceinline__ void m_two(const M3& p, const M3& q, M3& acc, M3& T) {
    if (P && Q) {
        T = acc + (p - q);
        acc = p + q;
    } else if (P) {
        T = acc + p;
        acc = p;
    } else if (Q) {
        T = acc - q;
        acc = q;
    }
}
// Corner values (0,0) (1,0) (0,1) (1,1) of plane sums T = (const, j, k, jk);
// HAS bit m: T[m] is not zero.
template <int HAS>
__device__ __forceinline__ void m_corners(const M3 (&T)[4], M3 (&f)[4]) {
    constexpr bool C = HAS & 1, Jm = HAS & 2, Km = HAS & 4, JK = HAS & 8;
    M3 a0{}, a1{}, b0{}, b1{};
    if (C && Km) { a0 = T[0] - T[2]; a1 = T[0] + T[2]; }
    else if (C) { a0 = T[0]; a1 = T[0]; }
    else if (Km) { a0 = -(T[2]); a1 = T[2]; }
    if (Jm && JK) { b0 = T[1] - T[3]; b1 = T[1] + T[3]; }
    else if (Jm) { b0 = T[1]; b1 = T[1]; }
    else if (JK) { b0 = -(T[3]); b1 = T[3]; }
    if ((C || Km) && (Jm || JK)) {
        f[0] = a0 - b0; f[1] = a0 + b0; f[2] = a1 - b1; f[3] = a1 + b1;
    } else if (C || Km) {
        f[0] = a0; f[1] = a0; f[2] = a1; f[3] = a1;
    } else {
        f[0] = -(b0); f[1] = b0; f[2] = -(b1); f[3] = b1;
    }
}

}  // namespace sordgpu
