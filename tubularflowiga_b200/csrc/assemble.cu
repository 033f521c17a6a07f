// FP64 VMS Navier-Stokes element assembly with the exact Newton tangent.
//
// Formulation: the reference's BuildNavierStokesElementFromPreparedPoints
// (solvers/cpu/include/NavierStokesElement.hpp:149-317, LegacyBodyFitted
// weak form, zero body force).  Its residual is the one the reference GPU
// kernel assembles (solvers/cuda/include/IgaCudaKernels.cuh:360-379); its
// tangent is the exact derivative (NavierStokesElement.hpp:244-312), not the
// frozen-tau tangent of the reference GPU kernel (IgaCudaKernels.cuh:380-396).
//
// Organisation.  Every term of the tangent is a product (test feature s of N_a) x (G_s of N_b) at a point
// (vms_tangent.cuh), so per row field i it is a matrix product over k = (point, s),
//   K^{if}_{ab} = sum_k G^{if}[(b, f)][k] Psi[k][a],   K = 64 points x 4 test features,
// and runs on the FP64 tensor path (mma.sync: operands in registers, so that shared memory serves
// three words per 64 products instead of one).  A CTA of 256 threads owns (element, row field, half of the
// functions b): 128 rows (b, f) x 64 functions a in registers, two CTAs per SM, so that one builds G while the
// other multiplies.  Per chunk of four points: G and Psi into padded shared buffers (one barrier a chunk), then
// the product.  m16n8k4 and not k16: scalar FP64 work of the builders queues behind the products on the same
// pipe, 32 cycles each instead of 128.  Rows, columns and CTAs past the element's own function
// count are skipped: elements at patch boundaries have 18 to 48 functions, and on the benchmark's meshes
// nen^2 is 40 to 65 % of 64^2.  The FP64 tensor pipe bounds it (55 % of its cycles on the cylinder; the rest are the
// latency of a warp's products and the barrier of a chunk).  The kernel it replaces (one CTA per SM, 8 x 8
// register tiles of scalar products over all 64 x 256 entries, the point state recomputed for each row
// field) took 34.5 ms for the 12,800-element section and 3.4 ms for the 1,280-element cylinder; this one takes
// 12.6 and 0.88 ms, 60 and 53 % of what the FP64 tensor pipe can do at the measured 63 products per cycle and SM.
#include "common.hpp"
#include "kernels.cuh"
#include "vms_point.cuh"
#include "vms_tangent.cuh"

namespace tfiga {
namespace {

constexpr int kThreads = 256;
constexpr int kChunkPoints = 4;                 // points per chunk
constexpr int kChunkK = kChunkPoints*4;         // depth of a chunk
constexpr int kHalf = 32;                       // functions b per CTA at most
// Strides (in doubles) that keep shared accesses free of bank conflicts: 16 lanes read 4 rows (fields of one
// function) x 4 columns of G and 4 x 4 of Psi; 8 lanes store 16 bytes each of eight functions.
constexpr int kGStride = kChunkK+4;
constexpr int kGFunction = 4*kGStride+2;
constexpr int kPsiStride = kMaxBasis+4;

struct AssembleShared {
	double G[2][kHalf*kGFunction];
	double Psi[3][kChunkK][kPsiStride];
	double pack[3][kChunkPoints][kPack];
};

__device__ __forceinline__ void Mma1684(double c[4], double a0, double a1, double b)
{
	asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
		: "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3]) : "d"(a0), "d"(a1), "d"(b));
}

struct PackReader {
	const double* p;
	__device__ __forceinline__ double operator()(int k) const { return p[k]; }
	__device__ __forceinline__ Two<double> two(int k) const
	{
		const double2 v = *reinterpret_cast<const double2*>(p+k);
		return {v.x, v.y};
	}
};

template <int I>
__device__ __forceinline__ void AssembleRow(AssembleShared& sm, const double* __restrict__ P,
	const double* __restrict__ packs, const int32_t* __restrict__ EB, int nen, int b0, int bn, double irho, double nu,
	double* __restrict__ values)
{
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int columns = (nen+7) & ~7;            // functions a in steps of eight
	// builder: a warp per (column-field pair, point), a lane per function b
	const int pair = warp >> 2, point = warp & 3;
	const bool builds = lane < bn;
	double ph[kFeatures];
	auto load = [&](int c) {
		if (builds) {
			const double* p = P+(size_t)(c*kChunkPoints+point)*kMaxBasis+b0+lane;
			#pragma unroll
			for (int t = 0; t < kFeatures; ++t) ph[t] = __ldg(p+(size_t)t*kQuad*kMaxBasis);
		}
	};
	auto stage = [&](int c, int slot) {
		// Psi rows k = 4 point + s, sixteen rows of up to 32 16-byte units, two rows per warp; the numbers
		#pragma unroll
		for (int r = 0; r < 2; ++r) {
			const int k = 2*warp+r;
			if (2*lane < columns) {
				const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.Psi[slot][k][2*lane]);
				const double* src = P+((size_t)(k & 3)*kQuad+c*kChunkPoints+(k >> 2))*kMaxBasis+2*lane;
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
			}
		}
		if (tid < kChunkPoints*kPack/2) {
			const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.pack[slot][0][0]+2*tid);
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst),
				"l"(packs+(size_t)c*kChunkPoints*kPack+2*tid) : "memory");
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	auto build = [&](int buffer, int slot) {
		if (!builds) return;
		const double* pk = sm.pack[slot][point];
		const PackReader coef{pk};
		const double n = ph[0], g[3] = {ph[1], ph[2], ph[3]};
		const double l = pk[kPackU]*g[0]+pk[kPackU+1]*g[1]+pk[kPackU+2]*g[2]-nu*ph[4];
		auto put = [&](int f, const double v[4]) {
			double2* d = reinterpret_cast<double2*>(&sm.G[buffer][lane*kGFunction+f*kGStride+4*point]);
			d[0] = make_double2(v[0], v[1]);
			d[1] = make_double2(v[2], v[3]);
		};
		double v[4];
		if (pair == 0) {
			TangentColumn<I, 0>(coef, n, g, l, irho, v);
			put(0, v);
			TangentColumn<I, 1>(coef, n, g, l, irho, v);
			put(1, v);
		} else {
			TangentColumn<I, 2>(coef, n, g, l, irho, v);
			put(2, v);
			TangentColumn<I, 3>(coef, n, g, l, irho, v);
			put(3, v);
		}
	};
	// The product's 16 x 8 tiles, row tile by row tile, in even runs over the eight warps: whole row tiles per
	// warp would leave two of the four schedulers half idle at 48 functions (six row tiles).
	constexpr int kTiles = kMaxBasis/8;          // tiles per warp at most
	const int across = columns >> 3, tiles = ((bn+3) >> 2)*across;
	const int tile0 = warp*tiles/8, mine = (warp+1)*tiles/8-tile0;
	const int m0 = tile0/across, n0 = tile0-m0*across;
	double acc[kTiles][4];
	#pragma unroll
	for (int t = 0; t < kTiles; ++t)
		#pragma unroll
		for (int k = 0; k < 4; ++k) acc[t][k] = 0.0;
	const int gr = lane >> 2, t4 = lane & 3;
	constexpr int kChunks = kQuad/kChunkPoints;
	load(0);
	stage(0, 0);
	stage(1, 1);
	asm volatile("cp.async.wait_group 1;" ::: "memory");
	__syncthreads();
	build(0, 0);
	load(1);
	for (int c = 0, slot = 0; c < kChunks; ++c) {
		const double* g_row = sm.G[c & 1]+(gr >> 2)*kGFunction+(gr & 3)*kGStride;
		const int buffer = c & 1, next = slot == 2 ? 0 : slot+1, after = next == 2 ? 0 : next+1;
		asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();                         // G of chunk c; numbers and Psi of chunk c + 1; chunk c - 1's are free
		if (c+2 < kChunks) stage(c+2, after);
		if (c+1 < kChunks) build(buffer^1, next);
		if (c+2 < kChunks) load(c+2);
		double a[8];
		int m = m0, n = n0;
		#pragma unroll
		for (int t = 0; t < kTiles; ++t)
			if (t < mine) {
				if (t == 0 || n == 0) {
					#pragma unroll
					for (int j = 0; j < 4; ++j) {
						a[2*j] = g_row[(4*m)*kGFunction+4*j+t4];
						a[2*j+1] = g_row[(4*m+2)*kGFunction+4*j+t4];
					}
				}
				double b[4];
				#pragma unroll
				for (int j = 0; j < 4; ++j) b[j] = sm.Psi[slot][4*j+t4][8*n+gr];
				#pragma unroll
				for (int j = 0; j < 4; ++j) Mma1684(acc[t], a[2*j], a[2*j+1], b[j]);
				if (++n == across) { n = 0; ++m; }
			}
		slot = next;
	}
	// rows gr and gr + 8 of row tile m are (function 4 m + gr / 4 [+ 2], field gr % 4), columns 8 n + 2 t4 [+ 1]
	// functions a: four lanes add one block row of a block, 32 contiguous bytes
	// (block indices fetched a tile ahead of the additions)
	auto blocks_of = [&](int m, int n, int out[4]) {
		#pragma unroll
		for (int u = 0; u < 4; ++u) {
			const int bl = 4*m+(gr >> 2)+2*(u >> 1), a = 8*n+2*t4+(u & 1);
			out[u] = a < nen && bl < bn ? __ldg(EB+a*kMaxBasis+b0+bl) : -1;
		}
	};
	int m = m0, n = n0, block[4];
	if (mine > 0) blocks_of(m, n, block);
	#pragma unroll
	for (int t = 0; t < kTiles; ++t)
		if (t < mine) {
			if (++n == across) { n = 0; ++m; }
			int ahead[4];
			if (t+1 < mine) blocks_of(m, n, ahead);
			#pragma unroll
			for (int u = 0; u < 4; ++u)
				if (block[u] >= 0) atomicAdd(values+(size_t)block[u]*16+I*4+(gr & 3), acc[t][u]);
			#pragma unroll
			for (int u = 0; u < 4; ++u) block[u] = ahead[u];
		}
}

__global__ void __launch_bounds__(kThreads, 2) AssembleKernel(DeviceMeshView mesh, int first,
	const double* __restrict__ phi, const double* __restrict__ packs, const int32_t* __restrict__ element_blocks,
	double irho, double nu, double* __restrict__ values)
{
	extern __shared__ __align__(16) unsigned char raw[];
	AssembleShared& sm = *reinterpret_cast<AssembleShared*>(raw);
	const int local = blockIdx.x >> 3, row = (blockIdx.x >> 1) & 3, half = blockIdx.x & 1;
	const int e = first+local;
	const int nen = mesh.element_offsets[e+1]-mesh.element_offsets[e];
	// the functions b in two even parts of whole row tiles, one part where 32 hold them all
	const int part = nen > kHalf ? (nen+7)/8*4 : nen;
	const int b0 = half*part, bn = min(part, nen-b0);
	if (bn <= 0) return;
	const double* P = phi+(size_t)e*kFeatures*kQuad*kMaxBasis;
	const double* pk = packs+(size_t)local*kQuad*kPack;
	const int32_t* EB = element_blocks+(size_t)e*kMaxBasis*kMaxBasis;
	if (row == 0) AssembleRow<0>(sm, P, pk, EB, nen, b0, bn, irho, nu, values);
	else if (row == 1) AssembleRow<1>(sm, P, pk, EB, nen, b0, bn, irho, nu, values);
	else if (row == 2) AssembleRow<2>(sm, P, pk, EB, nen, b0, bn, irho, nu, values);
	else AssembleRow<3>(sm, P, pk, EB, nen, b0, bn, irho, nu, values);
}

// Elements with 65..80 basis functions (rare: the spline extraction's extraordinary vertices), from
// their 80-wide tables.  CTA per (element, row field), 256 threads: nodal state, point state (warp per
// point), the row field's coefficients M_q and residual coefficients (thread per point), the residual
// (thread per basis function), then the tangent K^{if}_{ab} = sum_q sum_s Psi_s(a, q) sum_t
// M_q^{if}[s][t] Phi_t(b, q) with one task per (a, eight consecutive b): per point the task folds its
// test function into w[f][t] = sum_s Psi_s(a, q) M_q[f][s][t] and adds w[f][.] Phi_.(b, q) for its b.
// FP64 throughout; the sums are added into FP64 or FP32 block storage.
constexpr int kLargeThreads = 256;
constexpr int kLargeBGroup = 8;

constexpr size_t LargeSharedBytes()
{
	return sizeof(double)*(size_t)(kMaxBasisLarge*4*2+kQuad*kQS+kQuad*kCoef+kQuad*4);
}

template <class T>
__global__ void __launch_bounds__(kLargeThreads) AssembleLargeKernel(DeviceMeshView mesh, int first,
	const double* __restrict__ phi, const double* __restrict__ qdata, const int32_t* __restrict__ element_blocks,
	const double* __restrict__ state, const double* __restrict__ previous, AssemblyParams prm,
	T* __restrict__ values, double* __restrict__ rhs)
{
	constexpr int NP = kMaxBasisLarge;
	extern __shared__ __align__(16) double lsm[];
	double* U = lsm;                          // [NP][4]
	double* Up = U+NP*4;                      // [NP][4]
	double* QS = Up+NP*4;                     // [64][kQS]
	double* Msm = QS+kQuad*kQS;               // [64][kCoef]
	double* RC = Msm+kQuad*kCoef;             // [64][4]
	const int e = first+(blockIdx.x >> 2);
	const int row = blockIdx.x & 3;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int begin = mesh.element_offsets[e];
	const int nen = mesh.element_offsets[e+1]-begin;
	const double* P = phi+(size_t)(e-first)*kFeatures*kQuad*NP;

	for (int a = tid; a < NP; a += kLargeThreads) {
		double s[4] = {0.0, 0.0, 0.0, 0.0}, p[3] = {0.0, 0.0, 0.0};
		if (a < nen) {
			const size_t node = (size_t)mesh.connectivity[begin+a];
			for (int f = 0; f < 4; ++f) s[f] = state[4*node+f];
			if (prm.dt > 0.0) for (int f = 0; f < 3; ++f) p[f] = previous[4*node+f];
		}
		for (int f = 0; f < 4; ++f) U[a*4+f] = s[f];
		for (int f = 0; f < 3; ++f) Up[a*4+f] = p[f];
		Up[a*4+3] = 0.0;
	}
	__syncthreads();
	for (int q = warp; q < kQuad; q += kLargeThreads/32) {
		double v[22];
		#pragma unroll
		for (int k = 0; k < 22; ++k) v[k] = 0.0;
		for (int a = lane; a < NP; a += 32) {
			const double n = P[(0*kQuad+q)*NP+a];
			const double g0 = P[(1*kQuad+q)*NP+a], g1 = P[(2*kQuad+q)*NP+a], g2 = P[(3*kQuad+q)*NP+a];
			const double l = P[(4*kQuad+q)*NP+a];
			const double uf[4] = {U[a*4], U[a*4+1], U[a*4+2], U[a*4+3]};
			v[0] += n*uf[0]; v[1] += n*uf[1]; v[2] += n*uf[2]; v[3] += n*uf[3];
			v[4] += n*Up[a*4]; v[5] += n*Up[a*4+1]; v[6] += n*Up[a*4+2];
			#pragma unroll
			for (int f = 0; f < 4; ++f) { v[7+3*f] += g0*uf[f]; v[8+3*f] += g1*uf[f]; v[9+3*f] += g2*uf[f]; }
			v[19] += l*uf[0]; v[20] += l*uf[1]; v[21] += l*uf[2];
		}
		#pragma unroll
		for (int k = 0; k < 22; ++k)
			#pragma unroll
			for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
		if (lane == 0)
			#pragma unroll
			for (int k = 0; k < 22; ++k) QS[q*kQS+k] = v[k];
	}
	__syncthreads();
	if (tid < kQuad) {
		PointState S;
		const double* s = QS+tid*kQS;
		for (int c = 0; c < 3; ++c) {
			S.u[c] = s[kU+c]; S.up[c] = s[kUp+c]; S.lap[c] = s[kLap+c]; S.gp[c] = s[kGrad+9+c];
			for (int d = 0; d < 3; ++d) S.gv[c][d] = s[kGrad+3*c+d];
		}
		S.p = s[kP];
		RowCoefficients(row, S, qdata+((size_t)e*kQuad+tid)*kQData, prm, Msm+tid*kCoef, RC+tid*4);
	}
	__syncthreads();
	if (rhs != nullptr)
		for (int a = tid; a < nen; a += kLargeThreads) {
			double r = 0.0;
			for (int q = 0; q < kQuad; ++q)
				#pragma unroll
				for (int s = 0; s < 4; ++s) r += P[(s*kQuad+q)*NP+a]*RC[q*4+s];
			atomicAdd(rhs+4*(size_t)mesh.connectivity[begin+a]+row, r);
		}
	if (values == nullptr) return;
	const int32_t* EB = element_blocks+(size_t)(e-first)*NP*NP;
	constexpr int kGroups = NP/kLargeBGroup;
	for (int task = tid; task < NP*kGroups; task += kLargeThreads) {
		const int a = task/kGroups, b0 = (task%kGroups)*kLargeBGroup;
		if (a >= nen || b0 >= nen) continue;
		double acc[kLargeBGroup][4];
		#pragma unroll
		for (int j = 0; j < kLargeBGroup; ++j)
			#pragma unroll
			for (int f = 0; f < 4; ++f) acc[j][f] = 0.0;
		for (int q = 0; q < kQuad; ++q) {
			double psi[4];
			#pragma unroll
			for (int s = 0; s < 4; ++s) psi[s] = P[(s*kQuad+q)*NP+a];
			const double* Mq = Msm+q*kCoef;
			double w[4][5];
			#pragma unroll
			for (int f = 0; f < 4; ++f)
				#pragma unroll
				for (int t = 0; t < 5; ++t)
					w[f][t] = psi[0]*Mq[f*20+t]+psi[1]*Mq[f*20+5+t]+psi[2]*Mq[f*20+10+t]+psi[3]*Mq[f*20+15+t];
			#pragma unroll
			for (int j = 0; j < kLargeBGroup; ++j) {
				double ph[5];
				#pragma unroll
				for (int t = 0; t < 5; ++t) ph[t] = P[(t*kQuad+q)*NP+b0+j];
				#pragma unroll
				for (int f = 0; f < 4; ++f)
					acc[j][f] += w[f][0]*ph[0]+w[f][1]*ph[1]+w[f][2]*ph[2]+w[f][3]*ph[3]+w[f][4]*ph[4];
			}
		}
		#pragma unroll
		for (int j = 0; j < kLargeBGroup; ++j) {
			const int b = b0+j;
			if (b >= nen) break;
			const int block = EB[a*NP+b];
			if (block < 0) continue;
			T* dst = values+(size_t)block*16+row*4;
			#pragma unroll
			for (int f = 0; f < 4; ++f) atomicAdd(dst+f, (T)acc[j][f]);
		}
	}
}

} // namespace

void LaunchAssembleTangent(const DeviceMeshView& mesh, int first, int count, const double* phi, const double* packs,
	const int32_t* element_blocks, AssemblyParams params, double* values, cudaStream_t stream)
{
	if (count == 0) return;
	if (8LL*count > 0x7fffffffLL) Fail(-7, "too many elements for one assembly launch");
	CudaCheck(cudaFuncSetAttribute(AssembleKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)sizeof(AssembleShared)), "assembly shared-memory attribute");
	AssembleKernel<<<8u*(unsigned)count, kThreads, sizeof(AssembleShared), stream>>>(mesh, first, phi, packs,
		element_blocks, 1.0/params.density, params.viscosity/params.density, values);
	LaunchCheck("AssembleKernel");
}

template <class T>
void LaunchAssembleLarge(const DeviceMeshView& mesh, int first, int count, const double* phi, const double* qdata,
	const int32_t* element_blocks, const double* state, const double* previous, AssemblyParams params, T* values,
	double* rhs, cudaStream_t stream)
{
	if (count == 0 || (values == nullptr && rhs == nullptr)) return;
	constexpr size_t bytes = LargeSharedBytes();
	static bool configured = false;
	if (!configured) {
		CudaCheck(cudaFuncSetAttribute(AssembleLargeKernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
			(int)bytes), "large-element assembly shared-memory attribute");
		configured = true;
	}
	AssembleLargeKernel<T><<<4u*(unsigned)count, kLargeThreads, bytes, stream>>>(mesh, first, phi, qdata,
		element_blocks, state, previous, params, values, rhs);
	LaunchCheck("AssembleLargeKernel");
}

template void LaunchAssembleLarge<double>(const DeviceMeshView&, int, int, const double*, const double*,
	const int32_t*, const double*, const double*, AssemblyParams, double*, double*, cudaStream_t);
template void LaunchAssembleLarge<float>(const DeviceMeshView&, int, int, const double*, const double*,
	const int32_t*, const double*, const double*, AssemblyParams, float*, double*, cudaStream_t);

} // namespace tfiga
