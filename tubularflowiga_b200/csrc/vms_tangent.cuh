// The exact VMS tangent in factored form, shared by the FP64 and the tensor-core contraction.
//
// At a point every entry of the element tangent is a product of a test feature s of N_a (N, dN/dx, dN/dy,
// dN/dz) and a combination G_s of the trial function N_b (vms_point.cuh; NavierStokesElement.hpp:248-312).
// As a dense 4 x 5 coefficient matrix per pair of fields that is 320 numbers per point and 320 products per
// (b, point).  Collecting the terms by their common factors
//   L = u . grad N_b - nu Lap N_b   (the convection-diffusion operator of the strong residual),
//   A = a . grad N_b                (a = u + fine-scale velocity)
// leaves 72 numbers per point and about 130 products per (b, point) for all sixteen field pairs:
//   momentum row i, velocity column f:
//     G_0     = nn_if N - tg_if L + [i = f] rho A
//     G_{1+d} = c_ifd N + [i = f] (mu dN_d + pa_d L) + [d = i] rho tau_C dN_f + [d = f] (mu dN_i + pf_i L)
//   momentum row i, pressure column:
//     G_0 = -(1/rho) tg_i . grad N,   G_{1+d} = -[d = i] N + (1/rho) (pa_d dN_i + pf_i dN_d)
//   continuity row, velocity column f:  G_0 = dN_f,   G_{1+d} = -A_df N + [d = f] tau_M L
//   continuity row, pressure column:    G_0 = 0,      G_{1+d} = (tau_M / rho) dN_d
// All numbers carry the point's measure; those that are subtracted are stored negated, so that a column is
// multiplications and multiply-adds only.
//
// In FP32 (tensor-core modes) the numbers are rounded once from FP64 and a column's multiply-adds round again, a few
// 2^-24 beside the operands' own rounding (2^-17 split BF16, 2^-11 TF32, 2^-9 BF16).  Against coefficients formed in FP64
// and rounded once, the tangents' errors against FP64 are the same: over ten flows (steady, time steps of 1e-8 to 10 s,
// 0.2 and 20 m/s, viscosities of 3e-6 to 3.5 Pa s, a tube and a Y-bifurcation) the worst field pair's is 0.993 to 1.006
// of what it was in split BF16 (1.2e-6 to 3.0e-6), and 1.000 in TF32 and BF16.
#pragma once

#include "kernels.cuh"

namespace tfiga {

constexpr int kPack = kPointNumbers;             // numbers per point
// Ordered so that a column reads neighbours in pairs (every group starts at an even index).
enum : int {
	kPackColumn = 0,    // [6 (3 i + f)]: nn_if, -tg_if, c_if0, c_if1, c_if2, -A_if
	kPackU = 54,        // [e]  u_e (without the measure)
	kPackTau = 57,
	kPackRa = 58,       // [e]  rho a_e
	kPackMu = 61,
	kPackPa = 62,       // [d]  rho tau a_d
	kPackTauC = 65,     // rho tau_C
	kPackPf = 66,       // [i]  rho tau fine_i
	kPackOne = 69,      // measure
	kPackMinusOne = 70,
	kPackTauRho = 71
};

__device__ __forceinline__ double Fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double Mul(double a, double b) { return a*b; }

template <class V> struct Two {
	V a, b;
};

// G_0 .. G_3 of row field I and column field F.  coef(k): number k of the point, coef.two(k): numbers k and
// k + 1 (k even); g: gradient of N_b, l: L.  V: double, or a packed pair of floats with its own Fma and Mul.
template <int I, int F, class V, class Coef>
__device__ __forceinline__ void TangentColumn(const Coef& coef, V n, const V g[3], V l, V inverse_density, V out[4])
{
	if constexpr (I < 3 && F < 3) {
		constexpr int kColumn = kPackColumn+6*(3*I+F);
		const Two<V> nt = coef.two(kColumn), c01 = coef.two(kColumn+2), c2 = coef.two(kColumn+4);
		const Two<V> pt = coef.two(kPackPa+2), rm = coef.two(kPackRa+2);     // pa_2, tau_C; ra_2, mu
		const V c[3] = {c01.a, c01.b, c2.a}, pf = coef(kPackPf+I);
		out[0] = Fma(nt.a, n, Mul(nt.b, l));
		if constexpr (I == F) {
			const Two<V> ra = coef.two(kPackRa), pa = coef.two(kPackPa);
			const V p[3] = {pa.a, pa.b, pt.a};
			out[0] = Fma(ra.a, g[0], Fma(ra.b, g[1], Fma(rm.a, g[2], out[0])));
			#pragma unroll
			for (int d = 0; d < 3; ++d) out[1+d] = Fma(rm.b, g[d], Fma(p[d], l, Mul(c[d], n)));
			out[1+I] = Fma(pt.b, g[I], Fma(rm.b, g[I], Fma(pf, l, out[1+I])));
		} else {
			#pragma unroll
			for (int d = 0; d < 3; ++d) out[1+d] = Mul(c[d], n);
			out[1+I] = Fma(pt.b, g[F], out[1+I]);
			out[1+F] = Fma(rm.b, g[I], Fma(pf, l, out[1+F]));
		}
	} else if constexpr (I < 3) {
		const V pf = coef(kPackPf+I);
		const Two<V> pa = coef.two(kPackPa);
		const V p[3] = {pa.a, pa.b, coef(kPackPa+2)};
		out[0] = Mul(inverse_density, Fma(coef(kPackColumn+18*I+1), g[0],
			Fma(coef(kPackColumn+18*I+7), g[1], Mul(coef(kPackColumn+18*I+13), g[2]))));
		#pragma unroll
		for (int d = 0; d < 3; ++d) {
			const V w = Fma(p[d], g[I], Mul(pf, g[d]));
			out[1+d] = d == I ? Fma(inverse_density, w, Mul(coef(kPackMinusOne), n)) : Mul(inverse_density, w);
		}
	} else if constexpr (F < 3) {
		out[0] = Mul(coef(kPackOne), g[F]);
		#pragma unroll
		for (int d = 0; d < 3; ++d) {
			const V w = Mul(coef(kPackColumn+6*(3*d+F)+5), n);
			out[1+d] = d == F ? Fma(coef(kPackTau), l, w) : w;
		}
	} else {
		const V t = coef(kPackTauRho);
		out[0] = V{};
		#pragma unroll
		for (int d = 0; d < 3; ++d) out[1+d] = Mul(t, g[d]);
	}
}

} // namespace tfiga
