// State, residual and tangent numbers of every quadrature point, from one pass over the basis tables.
//
// Formulation: vms_point.cuh (residual) and vms_tangent.cuh (the tangent's numbers), FP64 throughout.
//
// What bounds it: the tables, 164 KB per element, read once.  A CTA of 128 threads owns an element and
// streams its points in eight chunks of eight (cp.async, the columns of the element's own functions only).
// Points need every function and the residual every point, so a chunk of points is the unit that reads each
// table entry once; the kernel it replaces read the tables twice and reduced 22 sums per point through
// shared memory.  Per chunk:
//   warp 0 forms the stabilisation, the residual's and the tangent's numbers, a lane per (point, row field),
//   a chain of some hundred dependent FP64 operations, while
//   warps 1 - 3 form the next chunk's state as a matrix product (8 points x functions x 8 fields per table)
//   on the FP64 tensor path, the functions split over the warps;
//   then all threads add the chunk's share of the residual, a thread per function and half of the points.
// Four CTAs per SM (54 KB of shared memory each) cover each other's latencies.
// 12,800-element section (nen 27 .. 64): 1225 us before; with the phases one after the other 660 us, now 547 us.
#include "common.hpp"
#include "kernels.cuh"
#include "vms_tangent.cuh"

#include <type_traits>

namespace tfiga {
namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads/32;
constexpr int kChunk = 8;                        // points per chunk
constexpr int kChunks = kQuad/kChunk;
constexpr int kRows = kFeatures*kChunk;          // table rows per chunk
constexpr int kSums = 64+4*32;                   // state sums of a chunk: 8 points x (8 fields of N, 4 of the rest)
constexpr int kStage = kPack+1;                  // row stride of a chunk's tangent numbers
constexpr int kSumWarps = kWarps-1;              // warps that form the next chunk's state

struct Shared {
	double ring[2][kRows][kMaxBasis];
	// state (4) and previous velocity (3) of every function, until the warps hold theirs; then the chunk's
	// tangent numbers, and at the end the residual of the second half of the points
	double stage[kChunk*kStage];
	double part[kSumWarps][kSums];
	double sums[kSums];
	double rc[kChunk][4][4];                     // [point][test feature][row field]
	double qd[2][kChunk*kQData];
};
static_assert(kMaxBasis*8 <= kChunk*kStage, "the functions' states fit the staged numbers' place");

// Entry a of a staged row: 16-byte units are swizzled by the point so that eight rows' equal columns lie in
// different banks.
__device__ __forceinline__ int Column(int point, int a)
{
	return (((a >> 1)^((point & 3) << 1)) << 1) | (a & 1);
}

__device__ __forceinline__ void Mma884(double& c0, double& c1, double a, double b)
{
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
		: "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}

// Material and time step with the quotients that every point uses (idt 0: steady).
struct PointParams {
	double rho, mu, nu, irho, idt;
};

// One (point, row field): residual numbers rc[test feature] and the row's tangent numbers into `pack`.
template <bool kTangent>
__device__ __forceinline__ void PointRow(int i, const double* sums, int q, const double* qd, const PointParams& prm,
	double rc[4], double* pack)
{
	const double rho = prm.rho, mu = prm.mu, nu = prm.nu, idt = prm.idt, irho = prm.irho;
	const double inverse_direction = 1.0/qd[7];
	double u[3], up[3], gv[3][3], gp[3], lap[3];
	#pragma unroll
	for (int c = 0; c < 3; ++c) {
		u[c] = sums[8*q+c];
		up[c] = sums[8*q+4+c];
		lap[c] = sums[64+96+4*q+c];
		gp[c] = sums[64+32*c+4*q+3];
		#pragma unroll
		for (int d = 0; d < 3; ++d) gv[c][d] = sums[64+32*d+4*q+c];
	}
	const double p = sums[8*q+3];
	const double meas = qd[0];
	const double G[3][3] = {{qd[1], qd[2], qd[3]}, {qd[2], qd[4], qd[5]}, {qd[3], qd[5], qd[6]}};
	double Gu[3], vm = 0.0, dudt[3];
	#pragma unroll
	for (int f = 0; f < 3; ++f) {
		Gu[f] = G[f][0]*u[0]+G[f][1]*u[1]+G[f][2]*u[2];
		vm += u[f]*Gu[f];
		dudt[f] = (u[f]-up[f])*idt;
	}
	// tau_M = S^(-1/2), tau_C = 1 / (tau_M |direction|^2) = S tau_M / |direction|^2
	const double S = 4.0*idt*idt+vm+(1.0/12.0)*nu*nu*qd[8];
	const double tau_m = rsqrt(S);
	const double tau_c = S*tau_m*inverse_direction;
	double R[3], fine[3], a[3];
	#pragma unroll
	for (int c = 0; c < 3; ++c) {
		R[c] = dudt[c]+u[0]*gv[c][0]+u[1]*gv[c][1]+u[2]*gv[c][2]+gp[c]*irho-nu*lap[c];
		fine[c] = -tau_m*R[c];
		a[c] = u[c]+fine[c];
	}
	const double divu = gv[0][0]+gv[1][1]+gv[2][2];
	// this lane's row of the velocity gradient, by selects (an index would put the array into local memory)
	const double fi = i == 0 ? fine[0] : i == 1 ? fine[1] : fine[2];
	double gi[3], gt[3];                             // du_i/dx_d and du_d/dx_i
	#pragma unroll
	for (int d = 0; d < 3; ++d) {
		gi[d] = i == 0 ? gv[0][d] : i == 1 ? gv[1][d] : gv[2][d];
		gt[d] = i == 0 ? gv[d][0] : i == 1 ? gv[d][1] : gv[d][2];
	}
	const double ti = i == 0 ? dudt[0] : i == 1 ? dudt[1] : dudt[2];
	if (i < 3) {
		rc[0] = -meas*(rho*(ti+a[0]*gi[0]+a[1]*gi[1]+a[2]*gi[2]));
		const double pressure = p-rho*tau_c*divu;
		#pragma unroll
		for (int d = 0; d < 3; ++d)
			rc[1+d] = -meas*(mu*(gi[d]+gt[d])-rho*fi*a[d]-(d == i ? pressure : 0.0));
	} else {
		rc[0] = -meas*divu;
		#pragma unroll
		for (int d = 0; d < 3; ++d) rc[1+d] = meas*fine[d];
	}
	if constexpr (!kTangent) return;
	// A[d][f] = -d(fine_d)/du_f without the gradient terms: tau^3 (G u)_f R_d - tau (idt delta + du_d/dx_f)
	const double t3 = tau_m*tau_m*tau_m;
	double A[3][3];
	#pragma unroll
	for (int d = 0; d < 3; ++d)
		#pragma unroll
		for (int f = 0; f < 3; ++f) A[d][f] = t3*Gu[f]*R[d]-tau_m*((d == f ? idt : 0.0)+gv[d][f]);
	const double mr = meas*rho;
	if (i < 3) {
		const double ui = i == 0 ? u[0] : i == 1 ? u[1] : u[2];
		const double ai = i == 0 ? a[0] : i == 1 ? a[1] : a[2];
		#pragma unroll
		for (int f = 0; f < 3; ++f) {
			const double Aif = i == 0 ? A[0][f] : i == 1 ? A[1][f] : A[2][f];
			double* column = pack+kPackColumn+6*(3*i+f);
			column[0] = mr*(gi[f]+(f == i ? idt : 0.0)+A[0][f]*gi[0]+A[1][f]*gi[1]+A[2][f]*gi[2]);
			column[1] = -mr*tau_m*gi[f];
			const double dtau_c = tau_c*tau_m*tau_m*Gu[f];
			#pragma unroll
			for (int d = 0; d < 3; ++d)
				column[2+d] = mr*((d == i ? dtau_c*divu : 0.0)-a[d]*Aif-fi*((d == f ? 1.0 : 0.0)+A[d][f]));
			column[5] = -meas*Aif;
		}
		pack[kPackPa+i] = mr*tau_m*ai;
		pack[kPackPf+i] = mr*tau_m*fi;
		pack[kPackU+i] = ui;
		pack[kPackRa+i] = mr*ai;
	} else {
		pack[kPackMu] = meas*mu;
		pack[kPackTauC] = mr*tau_c;
		pack[kPackOne] = meas;
		pack[kPackTau] = meas*tau_m;
		pack[kPackTauRho] = meas*tau_m*irho;
		pack[kPackMinusOne] = -meas;
	}
}

// Elements first + blockIdx.x.  packs (of C = float / double, null: none) start at element `first`: FP64
// [element][point][kPack], FP32 [element][point pair][kPack][2].
template <class C>
__global__ void __launch_bounds__(kThreads, 4) PointStreamKernel(DeviceMeshView mesh, int first,
	const double* __restrict__ phi, const double* __restrict__ qdata, const double* __restrict__ state,
	const double* __restrict__ previous, PointParams prm, C* __restrict__ packs, double* __restrict__ rhs)
{
	extern __shared__ __align__(16) unsigned char raw[];
	Shared& sm = *reinterpret_cast<Shared*>(raw);
	double* U = sm.stage;
	constexpr bool kTangent = !std::is_same<C, void>::value;
	const int e = first+blockIdx.x;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int begin = mesh.element_offsets[e];
	const int nen = mesh.element_offsets[e+1]-begin;
	const int columns = (nen+3) & ~3;                // the tables are zero past nen
	const double* P = phi+(size_t)e*kFeatures*kQuad*kMaxBasis;

	// Warps 1 - 3 fetch: they need the next chunk's rows while warp 0 is still with the last one's numbers.
	auto fetch = [&](int c, int buffer) {
		if (warp == 0) return;
		if (2*lane < columns) {
			#pragma unroll
			for (int r0 = 0; r0 < kRows; r0 += kSumWarps) {
				const int r = r0+warp-1, t = r/kChunk, q = r%kChunk;
				if (r < kRows) {
					const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.ring[buffer][r][Column(q, 2*lane)]);
					const double* src = P+((size_t)t*kQuad+c*kChunk+q)*kMaxBasis+2*lane;
					asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
				}
			}
		}
		if (tid-32 < kChunk*kQData/2) {
			const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.qd[buffer][2*(tid-32)]);
			const double* src = qdata+((size_t)e*kQuad+c*kChunk)*kQData+2*(tid-32);
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	fetch(0, 0);
	fetch(1, 1);

	if (tid < kMaxBasis) {
		double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
		if (tid < nen) {
			const size_t node = (size_t)mesh.connectivity[begin+tid];
			const double2 x01 = *reinterpret_cast<const double2*>(state+4*node);
			const double2 x23 = *reinterpret_cast<const double2*>(state+4*node+2);
			v[0] = x01.x; v[1] = x01.y; v[2] = x23.x; v[3] = x23.y;
			if (prm.idt > 0.0) {
				const double2 y01 = *reinterpret_cast<const double2*>(previous+4*node);
				v[4] = y01.x; v[5] = y01.y; v[6] = previous[4*node+2];
			}
		}
		#pragma unroll
		for (int f = 0; f < 8; ++f) U[tid*8+f] = v[f];
	}
	__syncthreads();
	// the functions of warps 1 - 3: steps of four, warp - 1, warp + 2, ...
	constexpr int kSteps = (kMaxBasis/4+kSumWarps-1)/kSumWarps;
	const int g = lane >> 2, t4 = lane & 3;
	const int steps = columns >> 2;
	double ub[kSteps];
	#pragma unroll
	for (int m = 0; m < kSteps; ++m) {
		const int s = warp-1+kSumWarps*m;
		ub[m] = warp > 0 && s < steps ? U[(4*s+t4)*8+g] : 0.0;
	}
	double res[4] = {0.0, 0.0, 0.0, 0.0};
	const int a = tid & 63, half = tid >> 6;

	auto form_state = [&](int buffer) {
		double acc[kFeatures][2];
		#pragma unroll
		for (int t = 0; t < kFeatures; ++t) acc[t][0] = acc[t][1] = 0.0;
		#pragma unroll
		for (int m = 0; m < kSteps; ++m) {
			const int s = warp-1+kSumWarps*m;
			if (s < steps) {
				#pragma unroll
				for (int t = 0; t < kFeatures; ++t)
					Mma884(acc[t][0], acc[t][1], sm.ring[buffer][t*kChunk+g][Column(g, 4*s+t4)], ub[m]);
			}
		}
		double* part = sm.part[warp-1];
		*reinterpret_cast<double2*>(&part[8*g+2*t4]) = make_double2(acc[0][0], acc[0][1]);
		if (t4 < 2) {
			#pragma unroll
			for (int t = 1; t < kFeatures; ++t)
				*reinterpret_cast<double2*>(&part[64+32*(t-1)+4*g+2*t4]) = make_double2(acc[t][0], acc[t][1]);
		}
	};
	auto add_parts = [&]() {
		for (int k = tid; k < kSums; k += kThreads) sm.sums[k] = (sm.part[0][k]+sm.part[1][k])+sm.part[2][k];
	};
	asm volatile("cp.async.wait_group 1;" ::: "memory");
	__syncthreads();
	if (warp > 0) form_state(0);
	__syncthreads();
	add_parts();
	__syncthreads();
	for (int c = 0; c < kChunks; ++c) {
		const int buffer = c & 1;
		if (warp == 0) {
			double rc[4];
			PointRow<kTangent>(t4, sm.sums, g, &sm.qd[buffer][g*kQData], prm, rc, sm.stage+g*kStage);
			#pragma unroll
			for (int s = 0; s < 4; ++s) sm.rc[g][s][t4] = rc[s];
		} else if (c+1 < kChunks) {
			asm volatile("cp.async.wait_group 0;" ::: "memory");
			asm volatile("bar.sync 1, %0;" :: "n"(32*kSumWarps) : "memory");   // chunk c + 1's rows
			form_state(buffer^1);
		}
		__syncthreads();
		if (rhs != nullptr && a < nen) {
			#pragma unroll
			for (int q = 0; q < kChunk/2; ++q) {
				const int point = half*(kChunk/2)+q;
				#pragma unroll
				for (int s = 0; s < 4; ++s) {
					const double psi = sm.ring[buffer][s*kChunk+point][Column(point, a)];
					const double2 r01 = *reinterpret_cast<const double2*>(&sm.rc[point][s][0]);
					const double2 r23 = *reinterpret_cast<const double2*>(&sm.rc[point][s][2]);
					res[0] = fma(psi, r01.x, res[0]); res[1] = fma(psi, r01.y, res[1]);
					res[2] = fma(psi, r23.x, res[2]); res[3] = fma(psi, r23.y, res[3]);
				}
			}
		}
		// a warp per two points
		if constexpr (std::is_same<C, double>::value) {
			double* out = packs+((size_t)blockIdx.x*kQuad+c*kChunk+2*warp)*kPack;
			const double* in = sm.stage+2*warp*kStage;
			for (int k = lane; k < kPack; k += 32) {
				out[k] = in[k];
				out[kPack+k] = in[kStage+k];
			}
		} else if constexpr (std::is_same<C, float>::value) {
			float2* out = reinterpret_cast<float2*>(packs+((size_t)blockIdx.x*kQuad+c*kChunk+2*warp)*kPack);
			const double* in = sm.stage+2*warp*kStage;
			for (int k = lane; k < kPack; k += 32) out[k] = make_float2((float)in[k], (float)in[kStage+k]);
		}
		if (c+1 < kChunks) add_parts();
		__syncthreads();                             // chunk c's rows and numbers are free, chunk c + 1's sums there
		if (c+2 < kChunks) fetch(c+2, buffer);
	}
	if (rhs == nullptr) return;
	// the two halves of the points, then into the nodes
	if (half == 1)
		#pragma unroll
		for (int f = 0; f < 4; ++f) sm.stage[4*a+f] = res[f];
	__syncthreads();
	if (half == 0 && a < nen) {
		double* r = rhs+4*(size_t)mesh.connectivity[begin+a];
		#pragma unroll
		for (int f = 0; f < 4; ++f) atomicAdd(r+f, res[f]+sm.stage[4*a+f]);
	}
}

template <class C>
void Launch(const DeviceMeshView& mesh, int first, int count, const double* phi, const double* qdata,
	const double* state, const double* previous, AssemblyParams params, C* packs, double* rhs, cudaStream_t stream)
{
	CudaCheck(cudaFuncSetAttribute(PointStreamKernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)sizeof(Shared)), "point kernel shared memory");
	const PointParams prm{params.density, params.viscosity, params.viscosity/params.density, 1.0/params.density,
		params.dt > 0.0 ? 1.0/params.dt : 0.0};
	PointStreamKernel<C><<<count, kThreads, sizeof(Shared), stream>>>(mesh, first, phi, qdata, state, previous, prm,
		packs, rhs);
	LaunchCheck("PointStreamKernel");
}

} // namespace

void LaunchPointStream(const DeviceMeshView& mesh, int first, int count, const double* phi, const double* qdata,
	const double* state, const double* previous, AssemblyParams params, double* packs64, float* packs32, double* rhs,
	cudaStream_t stream)
{
	if (count == 0) return;
	if (packs64) Launch<double>(mesh, first, count, phi, qdata, state, previous, params, packs64, rhs, stream);
	else if (packs32) Launch<float>(mesh, first, count, phi, qdata, state, previous, params, packs32, rhs, stream);
	else Launch<void>(mesh, first, count, phi, qdata, state, previous, params, nullptr, rhs, stream);
}

} // namespace tfiga
