// Device math for the SPH step engine: packed particle vectors, the cubic
// B-spline kernel, the reference's exact neighbor-range predicate and the
// Morton cell key. Every kernel is templated on the state precision R
// (float for production, double for the precision-study twin).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sph {

// 4-wide packed vector: {x, y, z, w}. The w lane carries a per-particle
// scalar that the same passes need (volume for positions, mass for
// velocities), so one 16-byte (f32) load brings both.
template <class R>
struct alignas(4 * sizeof(R)) R4 {
  R x, y, z, w;
};

// 2-wide packed pair (the second record of a sweep gather).
template <class R>
struct alignas(2 * sizeof(R)) R2 {
  R x, y;
};

template <class R>
struct V3 {
  R x, y, z;
};

template <class R>
__host__ __device__ __forceinline__ V3<R> v3(R x, R y, R z) { return {x, y, z}; }
template <class R>
__host__ __device__ __forceinline__ V3<R> xyz(const R4<R>& a) { return {a.x, a.y, a.z}; }
template <class R>
__host__ __device__ __forceinline__ V3<R> operator+(V3<R> a, V3<R> b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class R>
__host__ __device__ __forceinline__ V3<R> operator-(V3<R> a, V3<R> b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class R>
__host__ __device__ __forceinline__ V3<R> operator*(R s, V3<R> a) { return {s * a.x, s * a.y, s * a.z}; }
template <class R>
__host__ __device__ __forceinline__ V3<R>& operator+=(V3<R>& a, V3<R> b) { a.x += b.x; a.y += b.y; a.z += b.z; return a; }
template <class R>
__host__ __device__ __forceinline__ R dot(V3<R> a, V3<R> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <class R>
__host__ __device__ __forceinline__ V3<R> cross(V3<R> a, V3<R> b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// ---------------------------------------------------------------------------
// Cubic B-spline kernel (reference: simulation_lib/src/sph/kernel/mod.rs:17-46,
// kernel/cubic_spline.rs:7-17). h is the support radius; alpha = 16/pi.
//   W(r)    = alpha/h^3 * w(q),  w(q)  = (1-q)_+^3 - 4 (1/2-q)_+^3
//   gradW(r)= alpha/h^4 * r/|r| * w'(q), w'(q) = -3(1-q)_+^2 + 12 (1/2-q)_+^2
// ---------------------------------------------------------------------------
template <class R>
struct KernelConst {
  R h, inv_h, cw, cg;  // cw = alpha/h^3, cg = alpha/h^4
};

template <class R>
__host__ KernelConst<R> make_kernel_const(double h) {
  const double alpha = 16.0 / 3.14159265358979323846;
  KernelConst<R> k;
  k.h = (R)h;
  k.inv_h = (R)(1.0 / h);
  k.cw = (R)(alpha / (h * h * h));
  k.cg = (R)(alpha / (h * h * h * h));
  return k;
}

template <class R>
__device__ __forceinline__ R sq(R x) { return x * x; }

// a / b for the b > 0 of the pair loops. f32: the approximate reciprocal (an ulp) and one
// Newton step on the quotient, its residual in one fma. Before the last rounding the
// relative error is below 2^-45, so the result is the rounded quotient, or its neighbor
// where that lies within 2^-20 ulp of a tie.
__device__ __forceinline__ double quotient(double a, double b) { return a / b; }
__device__ __forceinline__ float quotient(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r;
  return fmaf(fmaf(-b, q, a), r, q);
}

// Two f32 operations in one instruction (each rounded like the scalar one).
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Both square roots, r0 and r1 > 0: r^2 rsqrt(r^2) and one Heron step, its residual in one
// fma. Before the last rounding the relative error is below 2^-43 (the approximate
// reciprocal root's is 2^-22.4 at most): the rounded root, or its neighbor where that lies
// within 2^-19 ulp of a tie.
__device__ __forceinline__ unsigned long long roots2(float r0, float r1) {
  float i0, i1;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(i0) : "f"(r0));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(i1) : "f"(r1));
  const unsigned long long d = pack2(r0, r1), inv = pack2(i0, i1);
  const unsigned long long r = mul2(d, inv);
  return fma2(fma2(mul2(r, pack2(-1.f, -1.f)), r, d), mul2(inv, pack2(0.5f, 0.5f)), r);
}

// W from the squared distance; zero outside the support.
template <class R>
__device__ __forceinline__ R kernel_w_r2(R r2, const KernelConst<R>& k) {
  R q = sqrt(r2) * k.inv_h;
  R a = q < R(1) ? R(1) - q : R(0);
  R b = q < R(0.5) ? R(0.5) - q : R(0);
  return k.cw * (a * a * a - R(4) * (b * b * b));
}

// Scalar factor f with gradW(r) = f * r (zero at r = 0 and outside support).
template <class R>
__device__ __forceinline__ R kernel_grad_factor(R r2, const KernelConst<R>& k) {
  if (!(r2 > R(0))) return R(0);
  R rn = sqrt(r2);
  R q = rn * k.inv_h;
  R a = q < R(1) ? R(1) - q : R(0);
  R b = q < R(0.5) ? R(0.5) - q : R(0);
  R dw = R(-3) * (a * a) + R(12) * (b * b);
  return k.cg * dw / rn;
}

// f32: w'(q) / |r| = 3 ((1-2q)_+^2 - (1-q)_+^2) / |r| from one approximate
// reciprocal square root; the clamps ride in saturating FMAs, and the squared
// distance is kept away from 0, where the factor is exactly 0, so that there is
// no compare and no select. The difference of squares cancels for close pairs, and
// (1-q)^2 has its own relative error near the support: relative to the factor, 1e-7
// (rms) for q in 0.3 to 0.6, 6e-7 at 0.1, 5e-6 at 0.01, 1.4e-6 at 0.9 (the form
// before, 12 (1/2-q)_+^2 - 3 (1-q)_+^2, cancels more). f64 keeps the exact form.
__device__ __forceinline__ float grad_third_r2(float r2, float inv_h) {  // -1/3 w'(q) / |r|, r2 > 0
  float inv, t, b;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(r2));
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(r2 * inv), "f"(-inv_h), "f"(1.f));  // (1-q)_+
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(b) : "f"(t), "f"(2.f), "f"(-1.f));           // (1-2q)_+
  return fmaf(-b, b, t * t) * inv;
}
template <>
__device__ __forceinline__ float kernel_grad_factor<float>(float r2, const KernelConst<float>& k) {
  return -3.f * k.cg * grad_third_r2(fmaxf(r2, 1e-30f), k.inv_h);
}

// The gradient factor without its constant, from the pair's offset: gradW(r) =
// -3 cg * grad_third * r. In f64 in its piecewise form, (2 - 3q) / h for
// q < 1/2 and (1-q)^2 / |r| beyond. The caller scales its sums by -3 cg once.
template <class R>
__device__ __forceinline__ R grad_third(R rx, R ry, R rz, R inv_h) {
  const R rn = sqrt(rx * rx + ry * ry + rz * rz);
  const R q = rn * inv_h;
  if (q < R(0.5)) return (R(2) - R(3) * q) * inv_h;
  const R t = R(1) - q;
  return q < R(1) ? t * t / rn : R(0);
}
// (1e-30 has no effect on any pair but the self pair)
template <>
__device__ __forceinline__ float grad_third<float>(float rx, float ry, float rz, float inv_h) {
  return grad_third_r2(fmaf(rz, rz, fmaf(ry, ry, fmaf(rx, rx, 1e-30f))), inv_h);
}

// The same for pass A of the sweeps, whose sums weigh close pairs most (p grows as they
// approach): for q < 1/3 in f32 the form without cancellation, (2 - 3q) / h, in one FMA on
// |r| = r^2 rsqrt(r^2) (rms relative error 2e-8 below 0.1, 5e-8 at 0.3); the two forms are
// equally exact at 1/3.
template <class R>
__device__ __forceinline__ R grad_third_close(R rx, R ry, R rz, R inv_h) {
  return grad_third(rx, ry, rz, inv_h);
}
template <>
__device__ __forceinline__ float grad_third_close<float>(float rx, float ry, float rz, float inv_h) {
  const float r2 = fmaf(rz, rz, fmaf(ry, ry, fmaf(rx, rx, 1e-30f)));
  float inv, t, b;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(r2));
  const float r = r2 * inv;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(t) : "f"(r), "f"(-inv_h), "f"(1.f));  // (1-q)_+
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(b) : "f"(t), "f"(2.f), "f"(-1.f));    // (1-2q)_+
  float f = fmaf(-b, b, t * t) * inv;
  // (predicated, which spares the select)
  asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, %2;\n\t@p fma.rn.f32 %0, %3, %4, %5;\n\t}"
      : "+f"(f) : "f"(t), "f"(2.f / 3.f), "f"(r), "f"(-3.f * inv_h * inv_h), "f"(2.f * inv_h));
  return f;
}

// Both W and the gradient factor from one square root.
template <class R>
__device__ __forceinline__ void kernel_w_and_grad(R r2, const KernelConst<R>& k, R& w, R& f) {
  R rn = sqrt(r2);
  R q = rn * k.inv_h;
  R a = q < R(1) ? R(1) - q : R(0);
  R b = q < R(0.5) ? R(0.5) - q : R(0);
  w = k.cw * (a * a * a - R(4) * (b * b * b));
  R dw = R(-3) * (a * a) + R(12) * (b * b);
  f = rn > R(0) ? k.cg * dw / rn : R(0);
}

// ---------------------------------------------------------------------------
// The reference's neighbor predicate, bit for bit: f64 difference of the two
// positions, squared norm summed as (dx^2 + dy^2) + dz^2 without contraction,
// IEEE sqrt, strict `< range` (spatial_hashing.rs:94, neighbor_search/mod.rs:31).
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool in_range_exact(double ax, double ay, double az, double bx,
                                               double by, double bz, double range) {
  double dx = __dsub_rn(ax, bx), dy = __dsub_rn(ay, by), dz = __dsub_rn(az, bz);
  double s = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return __dsqrt_rn(s) < range;
}

// Fast pre-filter in the state precision with a relative guard band; only
// pairs inside the band fall back to the exact f64 predicate. For R = float
// the f32 squared distance is within a few ulp of the exact value, far inside
// the 1e-5 band.
template <class R>
__device__ __forceinline__ bool in_range(const R4<R>& a, const R4<R>& b, double range,
                                         R range2_lo, R range2_hi) {
  R dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
  R r2 = dx * dx + dy * dy + dz * dz;
  if (r2 < range2_lo) return true;
  if (r2 > range2_hi) return false;
  return in_range_exact((double)a.x, (double)a.y, (double)a.z, (double)b.x, (double)b.y,
                        (double)b.z, range);
}

// Cell of a position: floor(p / cell_size) in f64, saturated to i32 like
// Rust's `as i32` (spatial_hashing.rs:40-46).
__device__ __forceinline__ int cell_coord(double p, double cell_size) {
  double f = floor(__ddiv_rn(p, cell_size));
  if (f != f) return 0;
  if (f >= 2147483647.0) return 2147483647;
  if (f <= -2147483648.0) return (int)0x80000000;
  return (int)f;
}

// Morton key of the low `bits` bits of each cell coordinate. Cells that wrap
// onto the same key share a bucket; the distance test separates them. Any
// two cells of one 3x3x3 stencil get distinct keys when bits >= 2.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  v &= 0x3ff;
  v = (v | (v << 16)) & 0x030000FF;
  v = (v | (v << 8)) & 0x0300F00F;
  v = (v | (v << 4)) & 0x030C30C3;
  v = (v | (v << 2)) & 0x09249249;
  return v;
}
__device__ __forceinline__ uint32_t morton_key(int cx, int cy, int cz, uint32_t mask) {
  return spread3((uint32_t)cx & mask) | (spread3((uint32_t)cy & mask) << 1) |
         (spread3((uint32_t)cz & mask) << 2);
}

// The inverse of spread3: every third bit of a key.
__device__ __forceinline__ uint32_t gather3(uint32_t v) {
  v &= 0x09249249;
  v = (v | (v >> 2)) & 0x030C30C3;
  v = (v | (v >> 4)) & 0x0300F00F;
  v = (v | (v >> 8)) & 0x030000FF;
  v = (v | (v >> 16)) & 0x3ff;
  return v;
}

// A particle's key in the spare lane of its position.
template <class R>
__device__ __forceinline__ R key_lane(uint32_t k);
template <>
__device__ __forceinline__ float key_lane<float>(uint32_t k) { return __uint_as_float(k); }
template <>
__device__ __forceinline__ double key_lane<double>(uint32_t k) { return __hiloint2double(0, (int)k); }
__device__ __forceinline__ uint32_t lane_key(float w) { return __float_as_uint(w); }
__device__ __forceinline__ uint32_t lane_key(double w) { return (uint32_t)__double2loint(w); }

}  // namespace sph
