// The exact VMS tangent in factored form, shared by the FP64 and the tensor-core contraction.
//
// At a point every entry of the element tangent is a product of a test feature s of N_a (N, dN/dx, dN/dy,
// dN/dz) and a combination G_s of the trial function N_b (vms_point.cuh; NavierStokesElement.hpp:248-312).
// As a dense 4 x 5 coefficient matrix per pair of fields that is 320 numbers per point and 320 products per
// (b, point).  Collecting the terms by their common factors
//   L = u . grad N_b - nu Lap N_b   (the convection-diffusion operator of the strong residual),
//   A = a . grad N_b                (a = u + fine-scale velocity)
// leaves 71 numbers per point and about 130 products per (b, point) for all sixteen field pairs:
//   momentum row i, velocity column f:
//     G_0     = nn_if N - tg_if L + [i = f] rho A
//     G_{1+d} = c_ifd N + [i = f] (mu dN_d + pa_d L) + [d = i] rho tau_C dN_f + [d = f] (mu dN_i + pf_i L)
//   momentum row i, pressure column:
//     G_0 = -(1/rho) tg_i . grad N,   G_{1+d} = -[d = i] N + (1/rho) (pa_d dN_i + pf_i dN_d)
//   continuity row, velocity column f:  G_0 = dN_f,   G_{1+d} = -A_df N + [d = f] tau_M L
//   continuity row, pressure column:    G_0 = 0,      G_{1+d} = (tau_M / rho) dN_d
// All numbers carry the point's measure.
#pragma once

#include "kernels.cuh"

namespace tfiga {

constexpr int kPack = kPointNumbers;             // numbers per point (one unused)
enum : int {
	kPackNN = 0,        // [3 i + f]
	kPackTg = 9,        // [3 i + f]  rho tau du_i/dx_f
	kPackC = 18,        // [9 i + 3 f + d]
	kPackPa = 45,       // [d]  rho tau a_d
	kPackPf = 48,       // [i]  rho tau fine_i
	kPackU = 51,        // [e]  u_e (without the measure)
	kPackRa = 54,       // [e]  rho a_e
	kPackMu = 57, kPackTauC = 58 /* rho tau_C */, kPackOne = 59 /* measure */, kPackTau = 60, kPackTauRho = 61,
	kPackA = 62         // [3 d + f]
};

// G_0 .. G_3 of row field I and column field F.  coef(k): number k of the point; g: gradient of N_b, l: L.
template <int I, int F, class V, class Coef>
__device__ __forceinline__ void TangentColumn(const Coef& coef, V n, const V g[3], V l, V inverse_density, V out[4])
{
	if constexpr (I < 3 && F < 3) {
		out[0] = coef(kPackNN+3*I+F)*n-coef(kPackTg+3*I+F)*l;
		if constexpr (I == F)
			out[0] = out[0]+coef(kPackRa)*g[0]+coef(kPackRa+1)*g[1]+coef(kPackRa+2)*g[2];
		#pragma unroll
		for (int d = 0; d < 3; ++d) {
			V v = coef(kPackC+9*I+3*F+d)*n;
			if (I == F) v = v+coef(kPackMu)*g[d]+coef(kPackPa+d)*l;
			if (d == I) v = v+coef(kPackTauC)*g[F];
			if (d == F) v = v+coef(kPackMu)*g[I]+coef(kPackPf+I)*l;
			out[1+d] = v;
		}
	} else if constexpr (I < 3) {
		const V t = coef(kPackTg+3*I)*g[0]+coef(kPackTg+3*I+1)*g[1]+coef(kPackTg+3*I+2)*g[2];
		out[0] = -inverse_density*t;
		#pragma unroll
		for (int d = 0; d < 3; ++d) {
			V v = inverse_density*(coef(kPackPa+d)*g[I]+coef(kPackPf+I)*g[d]);
			if (d == I) v = v-coef(kPackOne)*n;
			out[1+d] = v;
		}
	} else if constexpr (F < 3) {
		out[0] = coef(kPackOne)*g[F];
		#pragma unroll
		for (int d = 0; d < 3; ++d) {
			V v = -coef(kPackA+3*d+F)*n;
			if (d == F) v = v+coef(kPackTau)*l;
			out[1+d] = v;
		}
	} else {
		out[0] = V(0);
		#pragma unroll
		for (int d = 0; d < 3; ++d) out[1+d] = coef(kPackTauRho)*g[d];
	}
}

} // namespace tfiga
