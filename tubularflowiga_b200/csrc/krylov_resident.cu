// Restarted GMRES / flexible GMRES as one cooperative kernel, for systems whose Krylov basis fits the
// chip's shared memory (up to about 15,000 nodes at a restart of 64 in FP32).
//
// What bounds it.  On such systems the kernels of one Arnoldi step (scaled copy, AMG, SpMV, two
// Gram-Schmidt passes with their reductions, Givens) take 2 to 15 us each, mostly launch latency and
// ramp-up: on the 1,280-element cylinder an AMG-FGMRES step took 70 us in ten launches, for 29 MB of
// matrix that the L2 holds.  Here the CTAs (one per SM) stay resident for the whole solve.  Every CTA owns a
// contiguous range of block rows, balanced by blocks, and keeps its slice of the whole basis in shared
// memory, so both Gram-Schmidt passes read no memory beyond the partial sums; its work vector, the
// rotations and the Hessenberg column live there too.  A step then costs its SpMV, the AMG arrays and
// six grid barriers (three without AMG) of about 1.2 us.
//
// Phases of a step, a barrier after each: [restrict v_j | dense coarse solve | coarse correction and
// block-Jacobi: z_j |] SpMV of the own rows and first-pass dots | update and second-pass dots | update,
// v_{j+1} published, its norm.  Every CTA sums the others' partial sums itself in the same fixed order, so
// all of them take the same decisions without a broadcast, and results do not depend on timing.
//
// Independent segments (a batch of tubes) are groups of CTAs: each group has its own coefficients, norms,
// rotations and tolerance, and stops on its own; its CTAs then only take part in the barriers and the
// shared coarse solve.
//
// Memory written by other CTAs in this launch is read with plain (coherent after the barrier's acquire)
// loads, never through the read-only path.  Barrier waits are bounded: on expiry the status says so and
// every CTA returns.
#include "krylov_resident.hpp"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace tfiga {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads/32;
constexpr int kMaxRestart = 256;
constexpr int kMaxPieces = 4;
constexpr int kRestrictWarps = 8;              // warps per aggregate
constexpr int kDenseRows = 64;                 // coarse rows per CTA at most
constexpr unsigned long long kWaitNs = 4000000000ull;
constexpr int kIterationsPerLaunch = 4096;     // bounds one launch; a longer solve continues in the next

struct Args {
	ResidentProblem p;
	int restart, slice, pieces, ctas, groups;
	int max_cycles_iterations;
	const int32_t *cta_row, *cta_group, *group_cta, *agg_list, *agg_list_offsets;
	double *partial, *R, *y;
	const double* tolerance_in;                // a continued solve's tolerances, else null
	double* tolerance_out;
	int* flags;
	unsigned* barrier;
	ResidentStatus* status;
};

__device__ __forceinline__ double WarpSum(double v)
{
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

// Grid barrier on a counter that only grows; false when a wait ran out (in this or any CTA).
__device__ __forceinline__ bool GridBarrier(unsigned* counter, unsigned target, int* expired)
{
	__syncthreads();
	if (threadIdx.x == 0) {
		int bad = 0;
		asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(counter) : "memory");
		unsigned seen;
		unsigned long long start = 0;
		for (int spin = 0;; ++spin) {
			asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
			if (seen >= target) break;
			if ((spin & 255) == 255) {
				unsigned long long now;
				asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
				if (start == 0) start = now;
				else if (now-start > kWaitNs) { bad = 1; break; }
			}
		}
		__threadfence();
		if (bad) *expired = 1;
	}
	__syncthreads();
	return *expired == 0;
}

// Coherent loads of vectors that this launch writes.
__device__ __forceinline__ double2 Load2(const double* p)
{
	double2 v;
	asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
	return v;
}

// Lane's part of block row `row`, blocks first, first + step, ...: for 4x4 blocks four lanes share a
// block, one row each (a warp reads eight consecutive blocks at once, contiguously), so a row's sum needs
// three shuffles; for 2x2 blocks a lane takes a whole block.
template <int F, class T> struct RowPiece;

template <class T> struct BlockRow;
template <> struct BlockRow<float> {
	static __device__ __forceinline__ void Get(const float* v, size_t block, int r, double a[4])
	{
		const float4 q = __ldcs(reinterpret_cast<const float4*>(v+block*16+4*r));
		a[0] = q.x; a[1] = q.y; a[2] = q.z; a[3] = q.w;
	}
};
template <> struct BlockRow<double> {
	static __device__ __forceinline__ void Get(const double* v, size_t block, int r, double a[4])
	{
		const double2* q = reinterpret_cast<const double2*>(v+block*16+4*r);
		const double2 x = __ldg(q), y = __ldg(q+1);
		a[0] = x.x; a[1] = x.y; a[2] = y.x; a[3] = y.y;
	}
};

template <class T> struct RowPiece<4, T> {
	// the row sum r in lane r = 0 .. 3
	static __device__ __forceinline__ void Sum(const T* values, const int32_t* cols, const double* x, int lo, int hi,
		int lane, double out[1])
	{
		constexpr int kUnroll = sizeof(T) == 4 ? 4 : 2;
		const int r = lane & 3;
		double s = 0.0;
		int b = lo+(lane >> 2);
		for (; b+8*(kUnroll-1) < hi; b += 8*kUnroll) {
			int c[kUnroll];
			double a[kUnroll][4];
			#pragma unroll
			for (int u = 0; u < kUnroll; ++u) c[u] = __ldg(cols+b+8*u);
			#pragma unroll
			for (int u = 0; u < kUnroll; ++u) BlockRow<T>::Get(values, (size_t)(b+8*u), r, a[u]);
			#pragma unroll
			for (int u = 0; u < kUnroll; ++u) {
				const double2 p = Load2(x+4*(size_t)c[u]), q = Load2(x+4*(size_t)c[u]+2);
				s = fma(a[u][0], p.x, s); s = fma(a[u][1], p.y, s);
				s = fma(a[u][2], q.x, s); s = fma(a[u][3], q.y, s);
			}
		}
		for (; b < hi; b += 8) {
			const int c = __ldg(cols+b);
			double a[4];
			BlockRow<T>::Get(values, (size_t)b, r, a);
			const double2 p = Load2(x+4*(size_t)c), q = Load2(x+4*(size_t)c+2);
			s = fma(a[0], p.x, s); s = fma(a[1], p.y, s); s = fma(a[2], q.x, s); s = fma(a[3], q.y, s);
		}
		#pragma unroll
		for (int o = 16; o >= 4; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		out[0] = s;
	}
};

template <class T> struct RowPiece<2, T> {
	// the row sum r in lane r = 0, 1
	static __device__ __forceinline__ void Sum(const T* values, const int32_t* cols, const double* x, int lo, int hi,
		int lane, double out[1])
	{
		double s0 = 0.0, s1 = 0.0;
		#pragma unroll 2
		for (int b = lo+lane; b < hi; b += 32) {
			const int c = __ldg(cols+b);
			double a[4];
			if constexpr (sizeof(T) == 4) {
				const float4 q = __ldg(reinterpret_cast<const float4*>(values+4*(size_t)b));
				a[0] = q.x; a[1] = q.y; a[2] = q.z; a[3] = q.w;
			} else {
				const double2* q = reinterpret_cast<const double2*>(values+4*(size_t)b);
				const double2 u = __ldg(q), v = __ldg(q+1);
				a[0] = u.x; a[1] = u.y; a[2] = v.x; a[3] = v.y;
			}
			const double2 v = Load2(x+2*(size_t)c);
			s0 = fma(a[0], v.x, s0); s0 = fma(a[1], v.y, s0);
			s1 = fma(a[2], v.x, s1); s1 = fma(a[3], v.y, s1);
		}
		double keep = (lane & 1) ? s1 : s0;
		const double give = (lane & 1) ? s0 : s1;
		keep += __shfl_xor_sync(0xffffffffu, give, 1);
		#pragma unroll
		for (int o = 16; o >= 2; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
		out[0] = keep;
	}
};

template <class B> __device__ __forceinline__ double BasisLoad(const B* p)
{
	return (double)*reinterpret_cast<const volatile B*>(p);
}

template <int F, class T, class RT, class B, bool kFlex>
__global__ void __launch_bounds__(kThreads, 1) ResidentKrylovKernel(const Args a)
{
	extern __shared__ __align__(16) double sm[];
	__shared__ double red[kWarps][4];
	__shared__ double dense_part[kDenseRows][8];
	__shared__ double low_dot;
	__shared__ int expired;
	__shared__ double s_next;
	__shared__ int s_stop, s_all;
	const int m1 = a.restart+1;
	double* w = sm;                                    // [slice] work vector
	double* piece = w+a.slice;                         // [pieces * slice] SpMV pieces
	double* part = piece+(size_t)a.pieces*a.slice;     // [1024] update parts
	double* h = part+kThreads;                         // [restart + 1] this pass's coefficients
	double* col = h+m1;                                // [restart + 1] Hessenberg column
	double* scale = col+m1;
	double* cs = scale+m1;
	double* sn = cs+m1;
	double* g = sn+m1;
	double* pc = g+m1;                                 // rotation products
	double* tt = pc+m1;                                // rotation carries
	B* Vs = reinterpret_cast<B*>(tt+m1+(m1 & 1));      // [restart + 1][slice]

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int cta = blockIdx.x, G = a.ctas;
	const int row0 = a.cta_row[cta], row1 = a.cta_row[cta+1];
	const int lo = F*row0, len = F*(row1-row0);
	const int grp = a.cta_group[cta];
	const int g0 = a.group_cta[grp], g1 = a.group_cta[grp+1];
	const bool leader = cta == g0;
	const long long n = (long long)F*a.p.pattern.nodes;
	B* V = static_cast<B*>(a.p.V);
	double* R = a.R+(size_t)grp*a.restart*m1;          // rotated columns, contiguous
	double* y = a.y+(size_t)grp*m1;
	double* dots[2] = {a.partial, a.partial+(size_t)G*m1};
	double* norms = a.partial+(size_t)2*G*m1;
	unsigned epoch = 0;
	if (tid == 0) expired = 0;
	auto barrier = [&]() { ++epoch; return GridBarrier(a.barrier, epoch*(unsigned)G, &expired); };

	// Own rows of A v into `piece`, one warp per (row, piece of its blocks).
	auto product = [&](const auto* values, const double* x) {
		using VT = std::remove_cv_t<std::remove_pointer_t<decltype(values)>>;
		const int P = a.pieces, rows = row1-row0;
		for (int t = warp; t < rows*P; t += kWarps) {
			const int r = t/P, q = t-r*P;
			const int b0 = a.p.pattern.row_offsets[row0+r], b1 = a.p.pattern.row_offsets[row0+r+1];
			const int per = (b1-b0+P-1)/P;
			const int s0 = min(b1, b0+q*per), s1 = min(b1, s0+per);
			double v[1];
			RowPiece<F, VT>::Sum(values, a.p.pattern.columns, x, s0, s1, lane, v);
			if (lane < F) piece[(size_t)q*a.slice+F*r+lane] = v[0];
		}
	};
	auto piece_sum = [&](int k) {
		double s = piece[k];
		for (int q = 1; q < a.pieces; ++q) s += piece[(size_t)q*a.slice+k];
		return s;
	};
	// piece[0][k] += sum_k coef (g . x) g over the low-rank term's own entries; x global.
	auto low_rank = [&](const double* x) {
		for (int k = 0; k < a.p.low.count; ++k) {
			const int e0 = a.p.low.ptr[k], e1 = a.p.low.ptr[k+1];
			// entries are in ascending order: nothing to do for a CTA without any of them
			if (e0 >= e1 || a.p.low.idx[e1-1] < lo || a.p.low.idx[e0] >= lo+len) continue;
			double s = 0.0;
			for (int e = e0+tid; e < e1; e += kThreads)
				s = fma(a.p.low.val[e], *reinterpret_cast<const volatile double*>(x+a.p.low.idx[e]), s);
			s = WarpSum(s);
			if (lane == 0) red[warp][0] = s;
			__syncthreads();
			if (warp == 0) {
				const double t = WarpSum(red[lane][0]);
				if (lane == 0) low_dot = a.p.low.coef[k]*t;
			}
			__syncthreads();
			for (int e = e0+tid; e < e1; e += kThreads) {
				const int i = a.p.low.idx[e]-lo;
				if (i >= 0 && i < len) piece[i] = fma(low_dot, a.p.low.val[e], piece[i]);
			}
			__syncthreads();
		}
	};
	// w = [D^-1] scale (A x) of the own rows, from the pieces.
	auto finish_product = [&](double s, bool left) {
		for (int k = tid; k < len; k += kThreads) {
			double v;
			if (left) {
				const int r = k/F, c = k-r*F;
				const double* d = a.p.inverse+(size_t)(row0+r)*F*F+c*F;
				v = 0.0;
				#pragma unroll
				for (int f = 0; f < F; ++f) v = fma(d[f], s*piece_sum(r*F+f), v);
			} else {
				v = piece_sum(k);
			}
			w[k] = v;
		}
	};
	// partial sums scale_i <V_i, w> of the own slice: a warp per basis vector, or eight lanes where slices
	// are short.
	auto own_dots = [&](int count, double* out) {
		const int gw = len > 128 ? 32 : 8;
		const int per = 32/gw, sub = lane/gw, sl = lane%gw;
		for (int base = warp*per; base < count; base += kWarps*per) {
			const int i = base+sub;
			double s = 0.0;
			if (i < count) {
				const B* v = Vs+(size_t)i*a.slice;
				double t = 0.0;
				int k = sl;
				for (; k+gw < len; k += 2*gw) {
					s = fma((double)v[k], w[k], s);
					t = fma((double)v[k+gw], w[k+gw], t);
				}
				if (k < len) s = fma((double)v[k], w[k], s);
				s += t;
			}
			for (int o = gw >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
			if (sl == 0 && i < count) out[(size_t)i*G+cta] = s*scale[i];
		}
	};
	// h_i = sum of the group's partial sums; the column accumulates over the passes.
	auto gather_dots = [&](int count, const double* in, bool first) {
		for (int i = warp; i < count; i += 2*kWarps) {
			const int i2 = i+kWarps;
			const bool two = i2 < count;
			double s = 0.0, t = 0.0;
			for (int c = g0+lane; c < g1; c += 32) {
				s += *reinterpret_cast<const volatile double*>(in+(size_t)i*G+c);
				if (two) t += *reinterpret_cast<const volatile double*>(in+(size_t)i2*G+c);
			}
			s = WarpSum(s);
			t = WarpSum(t);
			if (lane == 0) {
				h[i] = s*scale[i];
				col[i] = first ? s : col[i]+s;
				if (two) {
					h[i2] = t*scale[i2];
					col[i2] = first ? t : col[i2]+t;
				}
			}
		}
	};
	// w -= sum_i h_i V_i on the own slice, the basis split over groups of threads.
	auto update = [&](int count) {
		const int width = (len+31)/32*32;
		const int parts = len == 0 ? 1 : max(1, min(16, kThreads/max(width, 1)));
		if (parts == 1) {
			for (int k = tid; k < len; k += kThreads) {
				double s0 = 0.0, s1 = 0.0;
				int i = 0;
				for (; i+1 < count; i += 2) {
					s0 = fma(h[i], (double)Vs[(size_t)i*a.slice+k], s0);
					s1 = fma(h[i+1], (double)Vs[(size_t)(i+1)*a.slice+k], s1);
				}
				if (i < count) s0 = fma(h[i], (double)Vs[(size_t)i*a.slice+k], s0);
				w[k] -= s0+s1;
			}
			return;
		}
		const int q = tid/width, k = tid-q*width;
		if (q < parts) {
			double s0 = 0.0, s1 = 0.0;
			if (k < len) {
				int i = q;
				for (; i+parts < count; i += 2*parts) {
					s0 = fma(h[i], (double)Vs[(size_t)i*a.slice+k], s0);
					s1 = fma(h[i+parts], (double)Vs[(size_t)(i+parts)*a.slice+k], s1);
				}
				if (i < count) s0 = fma(h[i], (double)Vs[(size_t)i*a.slice+k], s0);
			}
			part[tid] = s0+s1;
		}
		__syncthreads();
		if (tid < len) {
			double s = 0.0;
			for (int u = 0; u < parts; ++u) s += part[u*width+tid];
			w[tid] -= s;
		}
	};
	// The own slice of w becomes basis vector j (shared and global); this CTA's share of |w|^2.
	auto publish = [&](int j) {
		double sq = 0.0;
		for (int k = tid; k < len; k += kThreads) {
			const double v = w[k];
			Vs[(size_t)j*a.slice+k] = (B)v;
			V[(size_t)j*n+lo+k] = (B)v;
			sq = fma(v, v, sq);
		}
		sq = WarpSum(sq);
		if (lane == 0) red[warp][0] = sq;
		__syncthreads();
		if (warp == 0) {
			sq = WarpSum(red[lane][0]);
			if (lane == 0) norms[cta] = sq;
		}
	};
	auto group_norm = [&](int from, int to) {           // one warp; every lane gets the norm
		double s = 0.0;
		for (int c = from+lane; c < to; c += 32) s += *reinterpret_cast<const volatile double*>(norms+c);
		return sqrt(WarpSum(s));
	};
	// w = [D^-1] (rhs - A x) of the own rows
	auto residual = [&]() {
		product(static_cast<const RT*>(a.p.residual_values), a.p.x);
		__syncthreads();
		if (kFlex && a.p.low.count) low_rank(a.p.x);
		for (int k = tid; k < len; k += kThreads) w[k] = a.p.rhs[lo+k]-piece_sum(k);
		if (!kFlex) {
			__syncthreads();
			for (int k = tid; k < len; k += kThreads) piece[k] = w[k];
			__syncthreads();
			for (int k = tid; k < len; k += kThreads) {
				const int r = k/F, c = k-r*F;
				const double* d = a.p.inverse+(size_t)(row0+r)*F*F+c*F;
				double v = 0.0;
				#pragma unroll
				for (int f = 0; f < F; ++f) v = fma(d[f], piece[r*F+f], v);
				w[k] = v;
			}
		}
		__syncthreads();
	};
	auto report = [&](int converged, int iterations, int error, double res) {
		if (cta == 0 && tid == 0) {
			a.status->converged = converged;
			a.status->iterations = iterations;
			a.status->error = error;
			a.status->residual = res;
		}
	};
	auto give_up = [&](int iterations) {
		if (tid == 0) a.status->error = 4;
		if (cta == 0 && tid == 0) { a.status->converged = 0; a.status->iterations = iterations; }
	};

	int iterations = 0;
	double tolerance = 0.0;
	residual();
	publish(0);
	if (!barrier()) return give_up(iterations);
	for (int cycle = 0;; ++cycle) {
		// beta of the own group, then whether every group meets its tolerance (each CTA sums them all)
		const double beta = group_norm(g0, g1);
		if (cycle == 0) {
			tolerance = a.tolerance_in ? a.tolerance_in[grp] : fmax(a.p.tolerance_floor, a.p.rtol*beta);
			if (leader && tid == 0) a.tolerance_out[grp] = tolerance;
		}
		double total = 0.0;
		bool met = true, finite = true;
		if (a.groups == 1) {
			total = beta;
			finite = isfinite(beta);
			met = cycle == 0 && !a.tolerance_in ? beta == 0.0 : beta <= tolerance;
		} else {
			if (tid == 0) { s_all = 1; s_stop = 1; s_next = 0.0; }
			__syncthreads();
			// groups over warps; the tolerances of the others follow from their norms in the first cycle and
			// are read back afterwards (written before the last barriers)
			for (int q = warp; q < a.groups; q += kWarps) {
				const double b = group_norm(a.group_cta[q], a.group_cta[q+1]);
				const double tol = cycle == 0 && !a.tolerance_in ? fmax(a.p.tolerance_floor, a.p.rtol*b)
					: *reinterpret_cast<const volatile double*>(a.tolerance_in ? a.tolerance_in+q : a.tolerance_out+q);
				if (lane == 0) {
					if (!(b <= tol)) s_all = 0;
					if (!isfinite(b)) s_stop = 0;
					part[q] = b*b;
				}
			}
			__syncthreads();
			if (tid == 0) for (int q = 0; q < a.groups; ++q) s_next += part[q];
			__syncthreads();
			met = s_all != 0;
			finite = s_stop != 0;
			total = sqrt(s_next);
			__syncthreads();
		}
		if (!finite) return report(0, iterations, 2, total);
		if (met) return report(1, iterations, 0, total);
		if (iterations >= a.max_cycles_iterations || iterations >= a.p.max_iterations)
			return report(0, iterations, 0, total);
		const int cap = min(a.restart, a.p.max_iterations-iterations);
		bool open = a.groups == 1 || beta > tolerance;
		for (int i = tid; i <= a.restart; i += kThreads) { g[i] = 0.0; scale[i] = 0.0; }
		__syncthreads();
		if (tid == 0) {
			g[0] = beta;
			scale[0] = open && beta > 0.0 ? 1.0/beta : 0.0;
			if (leader) a.flags[grp] = open ? 0 : 1;
		}
		__syncthreads();
		int used = 0, j = 0;
		for (; j < cap; ++j) {
			if constexpr (kFlex) {
				// restriction of v_j: eight warps per aggregate of this CTA's list
				const int slots = kWarps/kRestrictWarps, slot = warp/kRestrictWarps;
				const int a0 = a.agg_list_offsets[cta], a1 = a.agg_list_offsets[cta+1];
				for (int base = a0; base < a1; base += slots) {
					const int which = base+slot;
					double acc[4] = {0.0, 0.0, 0.0, 0.0};
					if (which < a1 && open) {
						const int I = a.agg_list[which];
						const double s = scale[j];
						const int e1 = a.p.amg.agg_offsets[I+1];
						for (int k = a.p.amg.agg_offsets[I]+(tid & (32*kRestrictWarps-1)); k < e1; k += 32*kRestrictWarps) {
							const size_t i = 4*(size_t)a.p.amg.agg_order[k];
							const double2 m01 = *reinterpret_cast<const double2*>(a.p.amg.mask+i);
							const double2 m23 = *reinterpret_cast<const double2*>(a.p.amg.mask+i+2);
							const B* v = V+(size_t)j*n+i;
							acc[0] += m01.x*(s*BasisLoad(v)); acc[1] += m01.y*(s*BasisLoad(v+1));
							acc[2] += m23.x*(s*BasisLoad(v+2)); acc[3] += m23.y*(s*BasisLoad(v+3));
						}
					}
					#pragma unroll
					for (int c = 0; c < 4; ++c) {
						acc[c] = WarpSum(acc[c]);
						if (lane == 0) red[warp][c] = acc[c];
					}
					__syncthreads();
					if (tid < 4*slots) {
						const int q = base+tid/4;
						if (q < a1) {
							double s = 0.0;
							#pragma unroll
							for (int u = 0; u < kRestrictWarps; ++u) s += red[(tid/4)*kRestrictWarps+u][tid & 3];
							a.p.amg.coarse_rhs[4*(size_t)a.agg_list[q]+(tid & 3)] = s;
						}
					}
					__syncthreads();
				}
				if (!barrier()) return give_up(iterations);
				if (a.groups > 1) {
					// every group's flag was written before this barrier: all CTAs see the same
					if (warp == 0) {
						int still = 0;
						for (int q = lane; q < a.groups; q += 32)
							still |= *reinterpret_cast<const volatile int*>(a.flags+q) == 0;
						still = __any_sync(0xffffffffu, still);
						if (lane == 0) s_all = still ? 0 : 1;
					}
					__syncthreads();
					if (s_all) break;
				}
				// dense coarse solve: rows cta, cta + G, ..., each by `split` warps
				const int dn = 4*a.p.amg.coarse;
				const int mine = (dn-cta+G-1)/G;
				int split = 1;
				while (split < 8 && 2*split*mine <= kWarps && 64*split < dn) split *= 2;
				for (int t = warp; t < mine*split; t += kWarps) {
					const int k = t/split, q = t-k*split;
					const double2* ar = reinterpret_cast<const double2*>(a.p.amg.dense+(size_t)(cta+G*k)*a.p.amg.dense_ld);
					const int n2 = dn/2;
					double s = 0.0, u = 0.0;
					#pragma unroll 4
					for (int c = q*32+lane; c < n2; c += 32*split) {
						const double2 e = __ldg(ar+c), b = Load2(a.p.amg.coarse_rhs+2*c);
						s = fma(e.x, b.x, s);
						u = fma(e.y, b.y, u);
					}
					s = WarpSum(s+u);
					if (lane == 0) dense_part[k][q] = s;
				}
				__syncthreads();
				if (tid < mine) {
					double s = dense_part[tid][0];
					for (int q = 1; q < split; ++q) s += dense_part[tid][q];
					a.p.amg.coarse_x[cta+G*tid] = s;
				}
				if (!barrier()) return give_up(iterations);
				// z = P x_c + omega D^-1 (v - (A P) x_c), four lanes per node
				double* z = a.p.Z+(size_t)j*n;
				if (open) {
					const T* ap = static_cast<const T*>(a.p.amg.ap);
					const double s = scale[j];
					for (int k = tid; k < (len+31)/32*32; k += kThreads) {
						const int i = row0+(k >> 2), r = k & 3;
						const bool live = k < len;
						double v = 0.0;
						if (live) {
							v = s*(double)Vs[(size_t)j*a.slice+k];
							const int e1 = a.p.amg.ap_rows[i+1];
							for (int e = a.p.amg.ap_rows[i]; e < e1; ++e) {
								double b[4];
								BlockRow<T>::Get(ap, (size_t)e, r, b);
								const double* xc = a.p.amg.coarse_x+4*(size_t)a.p.amg.ap_cols[e];
								const double2 p = Load2(xc), q = Load2(xc+2);
								v -= b[0]*p.x+b[1]*p.y+b[2]*q.x+b[3]*q.y;
							}
						}
						const int base = lane & ~3;
						const double v0 = __shfl_sync(0xffffffffu, v, base), v1 = __shfl_sync(0xffffffffu, v, base+1);
						const double v2 = __shfl_sync(0xffffffffu, v, base+2), v3 = __shfl_sync(0xffffffffu, v, base+3);
						if (live) {
							const double2* d = reinterpret_cast<const double2*>(a.p.amg.inverse+(size_t)i*16+4*r);
							const double2 d01 = d[0], d23 = d[1];
							const double xc = *reinterpret_cast<const volatile double*>(
								a.p.amg.coarse_x+4*(size_t)a.p.amg.agg[i]+r);
							z[lo+k] = a.p.amg.mask[lo+k]*xc+a.p.amg.omega*(d01.x*v0+d01.y*v1+d23.x*v2+d23.y*v3);
						}
					}
				}
				if (!barrier()) return give_up(iterations);
				if (open) {
					product(static_cast<const T*>(a.p.krylov_values), z);
					__syncthreads();
					if (a.p.low.count) low_rank(z);
					finish_product(1.0, false);
				}
			} else {
				product(static_cast<const T*>(a.p.krylov_values), reinterpret_cast<const double*>(V)+(size_t)j*n);
				__syncthreads();
				finish_product(scale[j], true);
			}
			__syncthreads();
			const int count = j+1;
			if (open) own_dots(count, dots[0]);
			if (!barrier()) return give_up(iterations);
			if (open) {
				gather_dots(count, dots[0], true);
				__syncthreads();
				update(count);
				__syncthreads();
				own_dots(count, dots[1]);
			}
			if (!barrier()) return give_up(iterations);
			if (open) {
				gather_dots(count, dots[1], false);
				__syncthreads();
				update(count);
				__syncthreads();
				publish(j+1);
			}
			if (!barrier()) return give_up(iterations);
			if (open) {
				if (warp == 0) {
					// rotations of the new column: t_{i+1} = -s_i t_i + c_i h_{i+1} is the only serial part
					const double next = group_norm(g0, g1);
					if (lane == 0) col[j+1] = next;
					__syncwarp();
					for (int i = lane; i < j; i += 32) pc[i] = cs[i]*col[i+1];
					__syncwarp();
					if (lane == 0) {
						double t = col[0];
						#pragma unroll 8
						for (int i = 0; i < j; ++i) { tt[i] = t; t = fma(-sn[i], t, pc[i]); }
						const double mag = hypot(t, next);
						const double c = mag > 0.0 ? t/mag : 1.0, s = mag > 0.0 ? next/mag : 0.0;
						cs[j] = c; sn[j] = s;
						const double old = g[j];
						g[j] = c*old;
						g[j+1] = -s*old;
						const double res = fabs(g[j+1]);
						const int stop = res <= tolerance || next <= 1e-30;
						scale[j+1] = next > 1e-30 && !(stop && a.groups > 1) ? 1.0/next : 0.0;
						s_stop = stop;
						if (leader) {
							R[(size_t)j*m1+j] = mag;
							if (stop) a.flags[grp] = 1;
						}
					}
					__syncwarp();
					if (leader)
						for (int i = lane; i < j; i += 32) R[(size_t)j*m1+i] = fma(cs[i], tt[i], sn[i]*col[i+1]);
				}
				__syncthreads();
				used = j+1;
				if (s_stop) {
					open = false;
					if (a.groups == 1) { ++j; break; }
				}
			}
		}
		iterations += j;
		// least squares: back substitution by the leader's first warp, right-hand side in registers
		if (leader && warp == 0) {
			double b[kMaxRestart/32];
			#pragma unroll
			for (int q = 0; q < kMaxRestart/32; ++q) b[q] = 32*q+lane < used ? g[32*q+lane] : 0.0;
			for (int row = used-1; row >= 0; --row) {
				const double* c = R+(size_t)row*m1;
				double e[kMaxRestart/32];
				#pragma unroll
				for (int q = 0; q < kMaxRestart/32; ++q) e[q] = 32*q+lane <= row ? c[32*q+lane] : 0.0;
				double v = 0.0;
				#pragma unroll
				for (int q = 0; q < kMaxRestart/32; ++q)
					if (32*q+lane == row) {
						if (fabs(e[q]) < 1e-30) a.status->error = 1;
						else v = b[q]/e[q];
						y[row] = v;
					}
				v = __shfl_sync(0xffffffffu, v, row & 31);
				#pragma unroll
				for (int q = 0; q < kMaxRestart/32; ++q)
					if (32*q+lane < row) b[q] = fma(-e[q], v, b[q]);
			}
		}
		if (!barrier()) return give_up(iterations);
		if (*reinterpret_cast<const volatile int*>(&a.status->error) == 1) return report(0, iterations, 1, total);
		// x += sum_i y_i z_i (or y_i s_i v_i) on the own rows
		for (int i = tid; i < used; i += kThreads) {
			const double v = *reinterpret_cast<const volatile double*>(y+i);
			h[i] = kFlex ? v : v*scale[i];
		}
		__syncthreads();
		for (int k = tid; k < len; k += kThreads) {
			double v = a.p.x[lo+k];
			if constexpr (kFlex) {
				const double* z = a.p.Z+lo+k;
				#pragma unroll 4
				for (int i = 0; i < used; ++i) v = fma(h[i], z[(size_t)i*n], v);
			} else {
				for (int i = 0; i < used; ++i) v = fma(h[i], (double)Vs[(size_t)i*a.slice+k], v);
			}
			a.p.x[lo+k] = v;
		}
		if (!barrier()) return give_up(iterations);
		residual();
		publish(0);
		if (!barrier()) return give_up(iterations);
	}
}

using Kernel = void (*)(const Args);

Kernel KernelOf(ResidentKrylov::Kind kind)
{
	switch (kind) {
	case ResidentKrylov::kLeft2: return ResidentKrylovKernel<2, double, double, double, false>;
	case ResidentKrylov::kLeft2Fp32: return ResidentKrylovKernel<2, float, double, double, false>;
	case ResidentKrylov::kLeft4: return ResidentKrylovKernel<4, double, double, double, false>;
	case ResidentKrylov::kFlexDouble: return ResidentKrylovKernel<4, double, double, double, true>;
	case ResidentKrylov::kFlexFloat: return ResidentKrylovKernel<4, float, float, float, true>;
	default: return ResidentKrylovKernel<4, float, float, double, true>;
	}
}

} // namespace

ResidentKrylov::~ResidentKrylov()
{
	if (host_) cudaFreeHost(host_);
}

bool ResidentKrylov::Prepare(Kind kind, const DevicePatternView& pattern, int restart,
	const std::vector<int64_t>& segments, const AmgResidentView* amg, cudaStream_t stream)
{
	const long long version = amg ? amg->version : 0;
	if (planned_ && kind == kind_ && restart == restart_ && version == amg_version_ && segments == segments_)
		return fits_;
	kind_ = kind;
	restart_ = restart;
	amg_version_ = version;
	segments_ = segments;
	fits_ = false;
	Plan(pattern, amg, stream);
	planned_ = true;
	return fits_;
}

void ResidentKrylov::Plan(const DevicePatternView& pattern, const AmgResidentView* amg, cudaStream_t stream)
{
	const int fields = kind_ == kLeft2 || kind_ == kLeft2Fp32 ? 2 : 4;
	if (restart_ > kMaxRestart || pattern.nodes < 1) return;
	int device = 0, sms = 0, cooperative = 0, shared_max = 0;
	CudaCheck(cudaGetDevice(&device), "device");
	CudaCheck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "device attribute");
	CudaCheck(cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device), "device attribute");
	CudaCheck(cudaDeviceGetAttribute(&shared_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device), "device attribute");
	if (!cooperative) return;
	const Kernel kernel = KernelOf(kind_);
	cudaFuncAttributes attributes;
	CudaCheck(cudaFuncGetAttributes(&attributes, reinterpret_cast<const void*>(kernel)), "resident GMRES attributes");
	// the slice of an average CTA alone already says whether large systems fit
	const size_t entry = kind_ == kFlexFloat ? 4 : 8;
	if ((size_t)fields*pattern.nodes/sms*(restart_+1)*entry > (size_t)shared_max) return;
	std::vector<int32_t> rows((size_t)pattern.nodes+1);
	CudaCheck(cudaMemcpyAsync(rows.data(), pattern.row_offsets, rows.size()*sizeof(int32_t), cudaMemcpyDeviceToHost,
		stream), "row offsets");
	CudaCheck(cudaStreamSynchronize(stream), "row offsets");
	std::vector<int32_t> bounds;                     // node ranges of the groups
	if (segments_.empty()) bounds = {0, pattern.nodes};
	else for (const int64_t e : segments_) bounds.push_back((int32_t)(e/fields));
	groups_ = (int)bounds.size()-1;
	if (groups_ > sms) return;
	// one CTA per SM, fewer where a CTA would get less than about 100 KB of the matrix and 60 KB of basis; CTAs
	// over the groups by blocks, at least one each
	const long long blocks = rows[pattern.nodes];
	const long long basis = (long long)fields*pattern.nodes*(restart_+1)*(long long)entry;
	ctas_ = (int)std::min<long long>(sms, std::max<long long>({1, groups_, blocks/(fields == 4 ? 1024 : 4096),
		basis/60000}));
	std::vector<int> share(groups_, 1);
	for (int left = ctas_-groups_; left > 0; --left) {
		int best = 0;
		double most = -1.0;
		for (int q = 0; q < groups_; ++q) {
			const double load = (double)(rows[bounds[q+1]]-rows[bounds[q]])/share[q];
			if (load > most) { most = load; best = q; }
		}
		++share[best];
	}
	std::vector<int32_t> cta_row{0}, cta_group, group_cta{0};
	for (int q = 0; q < groups_; ++q) {
		// contiguous rows, balanced by blocks with a small constant per row
		const auto weight = [&](int r) { return (double)rows[r]+4.0*r; };
		const double base = weight(bounds[q]), all = weight(bounds[q+1])-base;
		int row = bounds[q];
		for (int c = 0; c < share[q]; ++c) {
			const double target = base+all*(c+1)/share[q];
			if (c+1 == share[q]) row = bounds[q+1];
			else while (row < bounds[q+1] && weight(row+1) <= target+0.5*(weight(row+1)-weight(row))) ++row;
			cta_row.push_back(row);
			cta_group.push_back(q);
		}
		group_cta.push_back((int32_t)cta_group.size());
	}
	int most_rows = 0;
	for (int c = 0; c < ctas_; ++c) most_rows = std::max(most_rows, cta_row[c+1]-cta_row[c]);
	// a slice stride of 8 modulo 16 entries spreads eight-lane dot groups over the banks
	slice_ = (fields*most_rows+15)/16*16+8;
	// split rows among warps until a CTA's last round of warps is a small part of its work
	pieces_ = 1;
	while (pieces_ < kMaxPieces && most_rows*pieces_ < 4*kWarps) pieces_ *= 2;
	if (fields == 2) pieces_ = 1;
	const size_t m1 = (size_t)restart_+1;
	smem_ = ((size_t)slice_*(1+pieces_)+kThreads+8*m1+(m1 & 1))*sizeof(double)+m1*slice_*entry;
	if (smem_+attributes.sharedSizeBytes > (size_t)shared_max) return;
	if (amg) {
		if (4*(long long)amg->coarse > (long long)ctas_*kDenseRows) return;
		if (groups_ > kThreads) return;
		// aggregates to CTAs of their own group, in turn
		std::vector<int32_t> of((size_t)pattern.nodes);
		CudaCheck(cudaMemcpyAsync(of.data(), amg->agg, of.size()*sizeof(int32_t), cudaMemcpyDeviceToHost, stream),
			"aggregates");
		CudaCheck(cudaStreamSynchronize(stream), "aggregates");
		std::vector<int32_t> group_of(amg->coarse, 0);
		for (int q = 0; q < groups_; ++q)
			for (int i = bounds[q]; i < bounds[q+1]; ++i) group_of[of[i]] = q;
		std::vector<std::vector<int32_t>> lists(ctas_);
		std::vector<int> turn(groups_, 0);
		for (int I = 0; I < amg->coarse; ++I) {
			const int q = group_of[I];
			lists[group_cta[q]+turn[q]++%share[q]].push_back(I);
		}
		std::vector<int32_t> list, offsets{0};
		for (const auto& l : lists) {
			list.insert(list.end(), l.begin(), l.end());
			offsets.push_back((int32_t)list.size());
		}
		agg_list_.Allocate(list.size());
		agg_list_.Upload(list.data(), list.size(), stream);
		agg_list_offsets_.Allocate(offsets.size());
		agg_list_offsets_.Upload(offsets.data(), offsets.size(), stream);
		CudaCheck(cudaStreamSynchronize(stream), "aggregate lists");
	}
	cta_row_.Allocate(cta_row.size());
	cta_row_.Upload(cta_row.data(), cta_row.size(), stream);
	cta_group_.Allocate(cta_group.size());
	cta_group_.Upload(cta_group.data(), cta_group.size(), stream);
	group_cta_.Allocate(group_cta.size());
	group_cta_.Upload(group_cta.data(), group_cta.size(), stream);
	partial_.Allocate((size_t)ctas_*(2*m1+1));
	R_.Allocate((size_t)groups_*restart_*m1);
	y_.Allocate((size_t)groups_*m1);
	tolerance_.Allocate((size_t)groups_);
	flags_.Allocate((size_t)groups_);
	status_.Allocate((sizeof(ResidentStatus)+3)/4);
	if (!host_) CudaCheck(cudaMallocHost(reinterpret_cast<void**>(&host_), sizeof(ResidentStatus)), "pinned status");
	CudaCheck(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)(shared_max-attributes.sharedSizeBytes)), "resident GMRES shared memory");
	int resident = 0;
	CudaCheck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, reinterpret_cast<const void*>(kernel), kThreads,
		smem_), "resident GMRES occupancy");
	CudaCheck(cudaStreamSynchronize(stream), "resident GMRES plan");
	fits_ = resident >= 1 && ctas_ <= sms;
}

ResidentStatus ResidentKrylov::Solve(const ResidentProblem& problem, cudaStream_t stream, long long* launches)
{
	Args args;
	args.p = problem;
	args.restart = restart_;
	args.slice = slice_;
	args.pieces = pieces_;
	args.ctas = ctas_;
	args.groups = groups_;
	args.max_cycles_iterations = kIterationsPerLaunch;
	args.cta_row = cta_row_.get();
	args.cta_group = cta_group_.get();
	args.group_cta = group_cta_.get();
	args.agg_list = agg_list_.get();
	args.agg_list_offsets = agg_list_offsets_.get();
	args.partial = partial_.get();
	args.R = R_.get();
	args.y = y_.get();
	args.tolerance_in = nullptr;
	args.tolerance_out = tolerance_.get();
	args.flags = flags_.get();
	args.status = reinterpret_cast<ResidentStatus*>(status_.get());
	args.barrier = &args.status->barrier;
	ResidentStatus total{};
	for (;;) {
		status_.Zero(stream);
		void* parameters[] = {&args};
		CudaCheck(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(KernelOf(kind_)), dim3(ctas_), dim3(kThreads),
			parameters, smem_, stream), "ResidentKrylovKernel");
		if (launches) *launches += 1;
		CudaCheck(cudaMemcpyAsync(host_, args.status, sizeof(ResidentStatus), cudaMemcpyDeviceToHost, stream),
			"resident GMRES status");
		CudaCheck(cudaStreamSynchronize(stream), "resident GMRES");
		total.converged = host_->converged;
		total.iterations += host_->iterations;
		total.error = host_->error;
		total.residual = host_->residual;
		if (total.error || total.converged || total.iterations >= problem.max_iterations || host_->iterations == 0)
			return total;
		args.tolerance_in = tolerance_.get();
		args.p.max_iterations = problem.max_iterations-total.iterations;
	}
}

} // namespace tfiga
