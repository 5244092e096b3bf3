// Fast form of the Gauss-point path for elastic stdBrick sets (the general meshes: distorted
// bricks, equalDOF ties, per-element materials): the point-parallel layout of points.cuh, built with
// fused multiply-adds. Each thread evaluates its point (shape functions, strain, stress, node forces,
// mass), and the points' 24 values are summed over the points in a fixed order (point 0 to 7), a
// thread per slot. The slot gather of general.cu then sums every equation in (element, DOF) order, as
// in the exact form, so the result is deterministic for any launch; it differs from the reference's
// arithmetic only by rounding (fused multiply-adds, per-point partial sums): within 1e-12 of the
// largest entry. The exact form (general.cu, no contraction) stays the parity mode.
#include "force.hpp"
#include "points.cuh"

namespace fx {
namespace {

using points::kEl;
using points::kThreads;

// Value a of the block's elements summed over the points, into its slots.
template <class S>
__device__ __forceinline__ void emit(const S& st, int32_t P, int32_t e, double* __restrict__ slots) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int a = w + 8 * k;
    double s = st.part[0][0][a][l];
#pragma unroll
    for (int g = 1; g < 8; ++g) s += st.part[g][0][a][l];
    slots[static_cast<int64_t>(a) * P + e] = s;
  }
}

// y_e = K_eff,e x_e (element_operator_apply, element_operator.hpp:82-130) for elastic sets.
__global__ void __launch_bounds__(kThreads, 2) k_apply_fast(const double* __restrict__ coords,
                                                         const int32_t* __restrict__ node,
                                                         const int32_t* __restrict__ eq,
                                                         const int32_t* __restrict__ param,
                                                         const ParamGP* __restrict__ params, int32_t N, int32_t P,
                                                         int32_t count, double ks, double kd, double km,
                                                         const double* __restrict__ x, double* __restrict__ slots,
                                                         const int* skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char raw[];
  auto& S = *reinterpret_cast<points::Stage<1, 1>*>(raw);
  points::stage_elements(S, coords, node, eq, N, P, count, x, nullptr);
  const int gp = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int32_t e = static_cast<int32_t>(blockIdx.x) * kEl + l;
  const bool ok = e < count;
  {
    const ParamGP& p = params[param[ok ? e : 0]];
    const OpFactors f = op_factors(p, ks, kd, km);
    const points::PointTable& tab = S.tab[gp];
    double dN[3][8], dvol, ep[6], sg[6];
    points::shape(S, tab, l, dN, dvol);
    points::strain(dN, S.x[0], l, ep);
    // elastic sets: D_eff = (cK + c0 + cc) D, D the isotropic matrix
    elastic_stress(p, ep, sg);
    const double c = (f.cK + f.c0 + f.cc) * dvol;
#pragma unroll
    for (int a = 0; a < 6; ++a) sg[a] *= c;
    const double cm = f.cM * (dvol * p.rho);
    double vg[3] = {0.0, 0.0, 0.0};
    if (cm != 0.0 && p.mass_type == 0)
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int q = 0; q < 3; ++q) vg[q] += tab.N[k] * S.x[0][3 * k + q][l];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      double fj[3];
      points::corner_force(dN, sg, j, fj);
      if (cm != 0.0) {
        const double t = cm * tab.N[j];
#pragma unroll
        for (int q = 0; q < 3; ++q) fj[q] += t * (p.mass_type == 0 ? vg[q] : S.x[0][3 * j + q][l]);
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) S.part[gp][0][3 * j + q][l] = fj[q];
    }
  }
  __syncthreads();
  if (ok) emit(S, P, e, slots);
}

// f_e = internal force + Rayleigh damping forces (StdBrick::compute_with, std_brick.hpp:492-543)
// for elastic sets: per point the stress and damping stress node forces, minus the body force,
// plus the alphaM mass force. The elastic tangent is the current, initial and committed one, so the
// damping stress is the stress of beta times the strain rate: one stress and one node force of the
// strain plus beta times the rate. DAMPED: a set has Rayleigh damping; undamped meshes stage no velocity
// (108 registers, not 124; B200, with the gather, against the damped form on them: 40^3 bricks 42.6 -> 39.0
// us, 48^3 65.8 -> 59.6, 75^3 256 -> 224).
template <bool DAMPED>
__global__ void __launch_bounds__(kThreads, 2) k_force_fast(const double* __restrict__ coords,
                                                         const int32_t* __restrict__ node,
                                                         const int32_t* __restrict__ eq,
                                                         const int32_t* __restrict__ param,
                                                         const ParamGP* __restrict__ params, int32_t N, int32_t P,
                                                         int32_t count, const double* __restrict__ u,
                                                         const double* __restrict__ v, double* __restrict__ slots) {
  extern __shared__ __align__(16) unsigned char raw[];
  auto& S = *reinterpret_cast<points::Stage<DAMPED ? 2 : 1, 1>*>(raw);
  points::stage_elements(S, coords, node, eq, N, P, count, u, v);
  const int gp = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int32_t e = static_cast<int32_t>(blockIdx.x) * kEl + l;
  const bool ok = e < count;
  {
    const ParamGP& p = params[param[ok ? e : 0]];
    const points::PointTable& tab = S.tab[gp];
    double dN[3][8], dvol, ep[6], sg[6];
    points::shape(S, tab, l, dN, dvol);
    points::strain(dN, S.x[0], l, ep);
    if constexpr (DAMPED) {
      const double beta = p.betaK + p.betaKinit + p.betaKcomm;
      if (beta != 0.0) {
        double rate[6];
        points::strain(dN, S.x[1], l, rate);
#pragma unroll
        for (int a = 0; a < 6; ++a) ep[a] += beta * rate[a];
      }
    }
    elastic_stress(p, ep, sg);
#pragma unroll
    for (int a = 0; a < 6; ++a) sg[a] *= dvol;
    double vg[3] = {0.0, 0.0, 0.0};
    if constexpr (DAMPED) {
      if (p.alphaM != 0.0 && p.mass_type == 0)
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int q = 0; q < 3; ++q) vg[q] += tab.N[k] * S.x[1][3 * k + q][l];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      double r[3];
      points::corner_force(dN, sg, j, r);
      const double t = tab.N[j] * dvol, am = p.alphaM * (t * p.rho);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        r[q] -= t * p.b[q];
        if constexpr (DAMPED)
          if (p.alphaM != 0.0) r[q] += am * (p.mass_type == 0 ? vg[q] : S.x[1][3 * j + q][l]);
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) S.part[gp][0][3 * j + q][l] = r[q];
    }
  }
  __syncthreads();
  if (ok) emit(S, P, e, slots);
}

unsigned fast_grid(int32_t count) { return static_cast<unsigned>((count + kEl - 1) / kEl); }

}  // namespace

bool general_fast_applies(const ForceState& s) {
  if (!s.fast_general) return false;
  for (const auto& p : s.params_h)
    if (p.kind != 0 || p.element != 0) return false;
  return true;
}

void general_apply_fast(ForceState& s, const double k[3], const double* x, double* y, cudaStream_t st, const int* skip) {
  static PerDevice<bool> set;
  allow_shared(set, k_apply_fast, sizeof(points::Stage<1, 1>));
  if (s.count > 0)
    k_apply_fast<<<fast_grid(s.count), kThreads, sizeof(points::Stage<1, 1>), st>>>(
        s.coords.ptr, s.node.ptr, s.eq.ptr, s.param.ptr, s.params.ptr, s.N, s.P, s.count, k[0], k[1], k[2], x,
        s.slots.ptr, skip);
  FX_LAUNCH_CHECK("element_apply_fast");
  general_gather(s, k, x, y, st, skip);
}

template <bool DAMPED>
static void launch_force_fast(ForceState& s, const double* u, const double* v, cudaStream_t st) {
  constexpr size_t bytes = sizeof(points::Stage<DAMPED ? 2 : 1, 1>);
  static PerDevice<bool> set;
  allow_shared(set, k_force_fast<DAMPED>, bytes);
  k_force_fast<DAMPED><<<fast_grid(s.count), kThreads, bytes, st>>>(s.coords.ptr, s.node.ptr, s.eq.ptr, s.param.ptr,
                                                                   s.params.ptr, s.N, s.P, s.count, u, v, s.slots.ptr);
}

void general_force_fast(ForceState& s, const double* u, const double* v, double* f, cudaStream_t st) {
  if (s.count > 0) {
    if (s.any_alpha || s.any_beta) launch_force_fast<true>(s, u, v, st);
    else launch_force_fast<false>(s, u, nullptr, st);
  }
  FX_LAUNCH_CHECK("element_force_fast");
  general_force_gather(s, v, f, st);
}

}  // namespace fx
