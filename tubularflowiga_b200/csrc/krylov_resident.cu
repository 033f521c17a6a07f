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
// five grid barriers (three without AMG) of 1.7 us.  Measured per step, separate launches against this kernel:
// cylinder, block-Jacobi FP64 GMRES(200) 68 -> 23 us, AMG-FGMRES FP64 70 -> 29 us; 12,800-element section, AMG-FGMRES
// FP32 105 -> 84 us (its 199 MB matrix streams from HBM), its transport GMRES(50) 58 -> 25 us; 6,176-element batch of
// five tubes 92 -> 35 us.
//
// Phases of a step, a barrier after each: [dense coarse solve | coarse correction and block-Jacobi: z_j |] SpMV of
// the own rows and first-pass dots | update and second-pass dots | update, v_{j+1} published with its norm and, for
// the coarse solve, every CTA's share of the aggregates' sums.  The rotations of a step run beside the next
// step's first phase.  Every CTA sums the others' partial sums itself in the same fixed order, so
// all of them take the same decisions without a broadcast, and results do not depend on timing.
//
// Independent segments (a batch of tubes) are groups of CTAs: each group has its own coefficients, norms,
// rotations and tolerance, and stops on its own; its CTAs then only take part in the barriers and the
// shared coarse solve.
//
// Memory written by other CTAs in this launch is read with plain (coherent after the barrier's acquire)
// loads, never through the read-only path.  Barrier waits are bounded (ResidentKrylov's wait limit): a CTA whose wait
// runs out says so in the status and returns, the others' waits run out in turn, and the caller solves by separate
// launches.
#include "krylov_resident.hpp"

#include "block_row.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace tfiga {
namespace {

// Threads per CTA: the flexible solves carry the AMG phases and gain from 128 registers (section step 51.9 ms in this
// kernel with 1024 threads, 47.3 with 512); the left-preconditioned ones spend most of a step on the Gram-Schmidt
// passes and gain from twice the threads (cylinder block-Jacobi solve 10.1 ms with 512, 9.4 with 1024).
constexpr int kThreadsFlexible = 512, kThreadsLeft = 1024;
constexpr int kMaxRestart = 256;
constexpr int kMaxPieces = 4;
constexpr int kDenseRows = 64;                 // coarse rows per CTA at most
constexpr int kCoarseMax = 512;                // aggregates at most (a coarse vector in shared memory)
// A matrix of at most this many bytes stays in the L2 (126 MB) from one product to the next, beside the vectors and the
// AMG's arrays; a larger one is loaded to leave the L2 first, so that the vectors stay.  (82 MB batch: 3.65 ms a solve
// streamed, 3.12 ms kept; 199 MB section: 7.75 ms streamed, 8.2 to 8.6 ms with 48 to 96 MB of it kept.)
constexpr size_t kKeepBytes = (size_t)96 << 20;

struct Args {
	ResidentProblem p;
	int restart, slice, pieces, ctas, groups;
	bool keep;                                 // the matrix stays in the L2
	int max_cycles_iterations;
	long long wait_ns;                         // limit of a barrier wait
	const int32_t *cta_row, *cta_group, *group_cta, *agg_list, *agg_list_offsets;
	// restriction: the nodes of every CTA by aggregate (part_nodes from part_start of its parts cta_parts ..), a
	// partial sum per part; each aggregate's parts are part_list from part_offsets; aggregates by group
	const int32_t *cta_parts, *part_start, *part_nodes, *part_offsets, *part_list, *group_agg, *group_agg_offsets;
	double* coarse_part;
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

// Grid barrier on a counter that only grows; false when this CTA's wait ran out (`expired` is the CTA's own: the others
// learn of it from their next wait).
__device__ __forceinline__ bool GridBarrier(unsigned* counter, unsigned target, long long wait_ns, int* expired)
{
	__syncthreads();
	if (threadIdx.x == 0) {
		int bad = 0;
		asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(counter) : "memory");
		unsigned seen;
		long long start = 0;
		for (int spin = 0;; ++spin) {
			asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
			if (seen >= target) break;
			if (wait_ns == 0) { bad = 1; break; }
			if ((spin & 255) == 255) {
				long long now;
				asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
				if (start == 0) start = now;
				else if (now-start > wait_ns) { bad = 1; break; }
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

// One piece of a block row, blocks lo .. hi - 1 (4x4: block_row.cuh; 2x2: a lane takes a whole block): the row sum r in
// lane r < F.
template <int F, class T, bool kStream>
__device__ __forceinline__ double PieceSum(const T* values, const int32_t* cols, const double* x, int lo, int hi,
	int lane)
{
	if constexpr (F == 4) {
		constexpr int kUnroll = sizeof(T) == 4 ? 4 : 2;
		const int r = lane & 3;
		double s = 0.0;
		int b = lo+(lane >> 2);
		for (; b+8*(kUnroll-1) < hi; b += 8*kUnroll) {
			int c[kUnroll];
			BlockRow<T> a[kUnroll];
			#pragma unroll
			for (int u = 0; u < kUnroll; ++u) c[u] = __ldg(cols+b+8*u);
			#pragma unroll
			for (int u = 0; u < kUnroll; ++u) a[u].template Load<kStream>(values, (size_t)(b+8*u), r);
			#pragma unroll
			for (int u = 0; u < kUnroll; ++u) s = a[u].Dot(Load2(x+4*(size_t)c[u]), Load2(x+4*(size_t)c[u]+2), s);
		}
		for (; b < hi; b += 8) {
			const int c = __ldg(cols+b);
			BlockRow<T> a;
			a.template Load<kStream>(values, (size_t)b, r);
			s = a.Dot(Load2(x+4*(size_t)c), Load2(x+4*(size_t)c+2), s);
		}
		return QuadRowSum(s);
	} else {
		double s0 = 0.0, s1 = 0.0;
		#pragma unroll 2
		for (int b = lo+lane; b < hi; b += 32) {
			const int c = __ldg(cols+b);
			double a[4];
			if constexpr (sizeof(T) == 4) {
				const float4 q = LoadMatrix<kStream>(reinterpret_cast<const float4*>(values+4*(size_t)b));
				a[0] = q.x; a[1] = q.y; a[2] = q.z; a[3] = q.w;
			} else {
				const double2* q = reinterpret_cast<const double2*>(values+4*(size_t)b);
				const double2 u = LoadMatrix<kStream>(q), v = LoadMatrix<kStream>(q+1);
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
		return keep;
	}
}

// Doubles that the own rows' offsets take (even, so that what follows stays 16-byte aligned).
__host__ __device__ constexpr int RowSlots(int slice, int fields) { return ((slice/fields+2)/2+2) & ~1; }

template <int F, class T, class RT, class B, bool kFlex>
__global__ void __launch_bounds__(kFlex ? kThreadsFlexible : kThreadsLeft, 1) ResidentKrylovKernel(const Args a)
{
	constexpr int kThreads = kFlex ? kThreadsFlexible : kThreadsLeft, kWarps = kThreads/32;
	extern __shared__ __align__(16) double sm[];
	__shared__ double red[kWarps];
	__shared__ double dense_part[kFlex ? kDenseRows : 1][8];
	__shared__ double low_dot;
	__shared__ int expired;
	__shared__ double s_next;
	__shared__ int s_stop, s_all;
	const int m1 = a.restart+1;
	double* w = sm;                                    // [slice] work vector
	double* piece = w+a.slice;                         // [pieces * slice] SpMV pieces
	double* part = piece+(size_t)a.pieces*a.slice;     // [kThreads] update parts
	double* h = part+kThreads;                         // [restart + 1] this pass's coefficients
	double* col = h+m1;                                // [restart + 1] Hessenberg column
	double* scale = col+m1;
	double* cs = scale+m1;
	double* sn = cs+m1;
	double* g = sn+m1;
	double* pc = g+m1;                                 // rotation products
	double* tt = pc+m1;                                // rotation carries
	int* rows = reinterpret_cast<int*>(tt+m1);          // [slice / F + 1] own row offsets
	double* coarse_b = tt+m1+RowSlots(a.slice, F);      // [4 coarse] the group's restricted vector (flexible)
	B* Vs = reinterpret_cast<B*>(coarse_b+(kFlex ? 4*kCoarseMax : 0));   // [restart + 1][slice]

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
	for (int r = tid; r <= row1-row0; r += kThreads) rows[r] = a.p.pattern.row_offsets[row0+r];
	__syncthreads();
	auto barrier = [&]() { ++epoch; return GridBarrier(a.barrier, epoch*(unsigned)G, a.wait_ns, &expired); };

	// Own rows of A x into `piece`, one warp per (row, piece of its blocks); warps `skip` and up take part.
	auto product = [&](const auto* values, const double* x, int skip, bool keep) {
		using VT = std::remove_cv_t<std::remove_pointer_t<decltype(values)>>;
		if (warp < skip) return;
		const int P = a.pieces, tasks = (row1-row0)*P, stride = kWarps-skip;
		const auto bounds = [&](int t, int& lo_, int& hi_) {
			const int r = t/P, q = t-r*P;
			const int b0 = rows[r], b1 = rows[r+1];
			const int per = (b1-b0+P-1)/P;
			lo_ = min(b1, b0+q*per);
			hi_ = min(b1, lo_+per);
		};
		for (int t = warp-skip; t < tasks; t += stride) {
			int b0, b1;
			bounds(t, b0, b1);
			const double v = keep
				? PieceSum<F, VT, false>(values, a.p.pattern.columns, x, b0, b1, lane)
				: PieceSum<F, VT, true>(values, a.p.pattern.columns, x, b0, b1, lane);
			if (lane < F) piece[(size_t)(t%P)*a.slice+F*(t/P)+lane] = v;
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
			if (lane == 0) red[warp] = s;
			__syncthreads();
			if (warp == 0) {
				const double t = WarpSum(lane < kWarps ? red[lane] : 0.0);
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
	// h_i = sum of the group's partial sums (several basis vectors per warp at a time, their loads in flight
	// together); the column accumulates over the passes.
	auto gather_dots = [&](int count, const double* in, bool first) {
		constexpr int kAtOnce = kFlex ? 4 : 2;
		for (int i = warp; i < count; i += kAtOnce*kWarps) {
			double s[kAtOnce];
			#pragma unroll
			for (int u = 0; u < kAtOnce; ++u) s[u] = 0.0;
			for (int c = g0+lane; c < g1; c += 32)
				#pragma unroll
				for (int u = 0; u < kAtOnce; ++u)
					if (i+u*kWarps < count)
						s[u] += *reinterpret_cast<const volatile double*>(in+(size_t)(i+u*kWarps)*G+c);
			#pragma unroll
			for (int u = 0; u < kAtOnce; ++u) {
				const int k = i+u*kWarps;
				if (k >= count) break;
				const double v = WarpSum(s[u]);
				if (lane == 0) {
					h[k] = v*scale[k];
					col[k] = first ? v : col[k]+v;
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
		if (lane == 0) red[warp] = sq;
		__syncthreads();
		if (warp == 0) {
			sq = WarpSum(lane < kWarps ? red[lane] : 0.0);
			if (lane == 0) norms[cta] = sq;
		}
		if constexpr (kFlex) {
			// the vector's share of every aggregate with nodes here: a warp per part, four lanes (fields) per node
			for (int k = a.cta_parts[cta]+warp; k < a.cta_parts[cta+1]; k += kWarps) {
				const int e1 = a.part_start[k+1];
				double s = 0.0;
				for (int e = a.part_start[k]+(lane >> 2); e < e1; e += 8) {
					const int i = 4*a.part_nodes[e]+(lane & 3);
					s = fma(a.p.amg.mask[i], (double)Vs[(size_t)j*a.slice+i-lo], s);
				}
				s = QuadRowSum(s);
				if (lane < 4) a.coarse_part[4*(size_t)k+lane] = s;
			}
		}
	};
	auto group_norm = [&](int from, int to) {           // one warp; every lane gets the norm
		double s = 0.0;
		for (int c = from+lane; c < to; c += 32) s += *reinterpret_cast<const volatile double*>(norms+c);
		return sqrt(WarpSum(s));
	};
	// w = [D^-1] (rhs - A x) of the own rows
	auto residual = [&]() {
		product(static_cast<const RT*>(a.p.residual_values), a.p.x, 0,
			a.keep && a.p.residual_values == a.p.krylov_values);
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
	// x as it was, for a caller who has to start again; kept by every CTA once the first barrier is passed, and x changes
	// only after that.  (The left-preconditioned solves are fewer and longer, and short of registers: the host keeps it.)
	if constexpr (kFlex)
		if (!a.tolerance_in)
			for (int k = tid; k < len; k += kThreads) a.p.start[lo+k] = a.p.x[lo+k];
	residual();
	publish(0);
	if (!barrier()) return give_up(iterations);
	if constexpr (kFlex)
		if (cta == 0 && tid == 0) a.status->kept = 1;
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
		// rotations of column j, by one warp: t_{i+1} = -s_i t_i + c_i h_{i+1} is the only serial part
		auto rotate = [&](int j) {
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
		};
		// Step j: the rotations of step j - 1 run in warp 0 beside the next thing that does not need them (the
		// coarse solve of the unscaled v_j, or its product); a stop discards that.
		int used = 0, j = 0;
		for (;; ++j) {
			const bool rotating = j > 0 && open;
			if (rotating && warp == 0) rotate(j-1);
			if constexpr (kFlex) {
				// the group's restricted v_j (unscaled) into shared memory: four threads per aggregate
				const int q0 = a.group_agg_offsets[grp], q1 = a.group_agg_offsets[grp+1];
				const int from = rotating ? 32 : 0;
				if (j < cap && tid >= from)
					for (int k = tid-from; k < 4*(q1-q0); k += kThreads-from) {
						const int I = a.group_agg[q0+(k >> 2)];
						const int e1 = a.part_offsets[I+1];
						double s = 0.0;
						#pragma unroll 4
						for (int e = a.part_offsets[I]; e < e1; ++e)
							s += *reinterpret_cast<const volatile double*>(a.coarse_part+4*(size_t)a.part_list[e]+(k & 3));
						coarse_b[k] = s;
					}
			} else {
				if (j < cap)
					product(static_cast<const T*>(a.p.krylov_values), reinterpret_cast<const double*>(V)+(size_t)j*n,
						rotating ? 1 : 0, a.keep);
			}
			__syncthreads();
			if (rotating) {
				used = j;
				if (s_stop) {
					open = false;
					if (a.groups == 1) break;
				}
			}
			if (j == cap) break;
			if constexpr (kFlex) {
				// dense coarse solve: the rows of this CTA's aggregates, each by `split` warps, over the group's columns
				const int l0 = a.agg_list_offsets[cta], mine = 4*(a.agg_list_offsets[cta+1]-l0);
				const int q0 = a.group_agg_offsets[grp], n2 = 2*(a.group_agg_offsets[grp+1]-q0);
				if (open) {
					int split = 1;
					while (split < 8 && 2*split*mine <= kWarps && 32*split < n2) split *= 2;
					for (int t = warp; t < mine*split; t += kWarps) {
						const int k = t/split, q = t-k*split;
						const double2* ar = reinterpret_cast<const double2*>(
							a.p.amg.dense+(size_t)(4*a.agg_list[l0+(k >> 2)]+(k & 3))*a.p.amg.dense_ld);
						double s = 0.0, u = 0.0;
						#pragma unroll 4
						for (int c = q*32+lane; c < n2; c += 32*split) {
							const double2 e = __ldg(ar+2*__ldg(a.group_agg+q0+(c >> 1))+(c & 1));
							const double2 b = *reinterpret_cast<const double2*>(coarse_b+2*c);
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
						a.p.amg.coarse_x[4*(size_t)a.agg_list[l0+(tid >> 2)]+(tid & 3)] = s*scale[j];
					}
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
				// z = P x_c + omega D^-1 (v - (A P) x_c), `lanes` per node (four rows, the A P blocks split over the
				// rest), x_c from shared memory
				double* z = a.p.Z+(size_t)j*n;
				if (open) {
					for (int k = tid; k < 2*a.p.amg.coarse; k += kThreads)
						reinterpret_cast<double2*>(coarse_b)[k] = Load2(a.p.amg.coarse_x+2*k);
					__syncthreads();
					const T* ap = static_cast<const T*>(a.p.amg.ap);
					const double s = scale[j];
					int lanes = 4;
					while (lanes < 32 && 2*lanes*(row1-row0) <= kThreads) lanes *= 2;
					const int r = lane & 3, sub = (lane%lanes) >> 2, step = lanes >> 2;
					for (int k = tid; k < ((row1-row0)*lanes+31)/32*32; k += kThreads) {
						const int node = k/lanes, i = row0+node;
						const bool live = node < row1-row0;
						double v = 0.0;
						if (live) {
							const int e1 = a.p.amg.ap_rows[i+1];
							constexpr int kAtOnce = 4;
							for (int e = a.p.amg.ap_rows[i]+sub; e < e1; e += kAtOnce*step) {
								BlockRow<T> b[kAtOnce];
								int c[kAtOnce];
								#pragma unroll
								for (int u = 0; u < kAtOnce; ++u) {
									const int at = min(e+u*step, e1-1);
									c[u] = __ldg(a.p.amg.ap_cols+at);
									b[u].template Load<false>(ap, (size_t)at, r);
								}
								#pragma unroll
								for (int u = 0; u < kAtOnce; ++u) {
									const double2* xc = reinterpret_cast<const double2*>(coarse_b+4*c[u]);
									if (e+u*step < e1) v -= b[u].Dot(xc[0], xc[1], 0.0);
								}
							}
						}
						for (int o = lanes >> 1; o >= 4; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
						if (live) v = fma(s, (double)Vs[(size_t)j*a.slice+4*node+r], v);
						const int base = lane & ~3;
						const double v0 = __shfl_sync(0xffffffffu, v, base), v1 = __shfl_sync(0xffffffffu, v, base+1);
						const double v2 = __shfl_sync(0xffffffffu, v, base+2), v3 = __shfl_sync(0xffffffffu, v, base+3);
						if (live && sub == 0) {
							const double2* d = reinterpret_cast<const double2*>(a.p.amg.inverse+(size_t)i*16+4*r);
							const double2 d01 = d[0], d23 = d[1];
							const size_t at = 4*(size_t)i+r;
							z[at] = a.p.amg.mask[at]*coarse_b[4*a.p.amg.agg[i]+r]
								+a.p.amg.omega*(d01.x*v0+d01.y*v1+d23.x*v2+d23.y*v3);
						}
					}
				}
				if (!barrier()) return give_up(iterations);
				if (open) {
					product(static_cast<const T*>(a.p.krylov_values), z, 0, a.keep);
					__syncthreads();
					if (a.p.low.count) low_rank(z);
					finish_product(1.0, false);
				}
			} else {
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
	try {
		Plan(pattern, amg, stream);
	} catch (const Error&) {
		// no memory for the work arrays or the kernel's code: the separate launches need neither
		ReleaseArrays();
		fits_ = false;
	}
	planned_ = true;
	return fits_;
}

void ResidentKrylov::ReleaseArrays()
{
	for (auto* a : {&cta_row_, &cta_group_, &group_cta_, &agg_list_, &agg_list_offsets_, &status_}) a->Release();
	for (auto& a : tables_) a.Release();
	for (auto* a : {&partial_, &R_, &y_, &tolerance_, &coarse_part_}) a->Release();
	flags_.Release();
}

void ResidentKrylov::Plan(const DevicePatternView& pattern, const AmgResidentView* amg, cudaStream_t stream)
{
	const int fields = kind_ == kLeft2 || kind_ == kLeft2Fp32 ? 2 : 4;
	threads_ = amg ? kThreadsFlexible : kThreadsLeft;
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
	const size_t value_bytes = fields == 4 ? (kind_ == kLeft4 || kind_ == kFlexDouble ? 128 : 64)
		: kind_ == kLeft2 ? 32 : 16;
	keep_ = (size_t)blocks*value_bytes <= kKeepBytes;
	int most_rows = 0;
	for (int c = 0; c < ctas_; ++c) most_rows = std::max(most_rows, cta_row[c+1]-cta_row[c]);
	// a slice stride of 8 modulo 16 entries spreads eight-lane dot groups over the banks
	slice_ = (fields*most_rows+15)/16*16+8;
	// split rows among warps until a CTA's last round of warps is a small part of its work
	pieces_ = 1;
	while (pieces_ < kMaxPieces && most_rows*pieces_ < threads_/8) pieces_ *= 2;
	if (fields == 2) pieces_ = 1;
	const size_t m1 = (size_t)restart_+1;
	smem_ = ((size_t)slice_*(1+pieces_)+threads_+8*m1+RowSlots(slice_, fields)
		+(amg ? 4*(size_t)kCoarseMax : 0))*sizeof(double)+m1*slice_*entry;
	if (smem_+attributes.sharedSizeBytes > (size_t)shared_max) return;
	if (groups_ > threads_) return;
	if (amg) {
		if (amg->coarse > kCoarseMax) return;
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
			if (4*l.size() > (size_t)kDenseRows) return;
			list.insert(list.end(), l.begin(), l.end());
			offsets.push_back((int32_t)list.size());
		}
		std::vector<int32_t> group_agg, group_agg_offsets{0};
		for (int q = 0; q < groups_; ++q) {
			for (int I = 0; I < amg->coarse; ++I)
				if (group_of[I] == q) group_agg.push_back(I);
			group_agg_offsets.push_back((int32_t)group_agg.size());
		}
		// every CTA's nodes by aggregate, and every aggregate's parts in the order of the CTAs
		std::vector<int32_t> cta_parts{0}, part_start, part_nodes, part_agg;
		for (int c = 0; c < ctas_; ++c) {
			std::vector<int32_t> nodes(cta_row[c+1]-cta_row[c]);
			for (size_t k = 0; k < nodes.size(); ++k) nodes[k] = cta_row[c]+(int32_t)k;
			std::stable_sort(nodes.begin(), nodes.end(), [&](int32_t x, int32_t y) { return of[x] < of[y]; });
			for (size_t k = 0; k < nodes.size(); ++k) {
				if (k == 0 || of[nodes[k]] != of[nodes[k-1]]) {
					part_start.push_back((int32_t)part_nodes.size());
					part_agg.push_back(of[nodes[k]]);
				}
				part_nodes.push_back(nodes[k]);
			}
			cta_parts.push_back((int32_t)part_start.size());
		}
		part_start.push_back((int32_t)part_nodes.size());
		std::vector<int32_t> part_offsets(amg->coarse+1, 0), part_list(part_agg.size());
		for (const int32_t I : part_agg) ++part_offsets[I+1];
		for (int I = 0; I < amg->coarse; ++I) part_offsets[I+1] += part_offsets[I];
		std::vector<int32_t> fill(part_offsets.begin(), part_offsets.end()-1);
		for (size_t k = 0; k < part_agg.size(); ++k) part_list[fill[part_agg[k]]++] = (int32_t)k;
		const std::vector<int32_t>* tables[] = {&cta_parts, &part_start, &part_nodes, &part_offsets, &part_list, &group_agg,
			&group_agg_offsets};
		for (int k = 0; k < kTables; ++k) {
			tables_[k].Allocate(tables[k]->size());
			tables_[k].Upload(tables[k]->data(), tables[k]->size(), stream);
		}
		coarse_part_.Allocate(4*part_agg.size());
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
	CudaCheck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, reinterpret_cast<const void*>(kernel), threads_,
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
	args.keep = keep_;
	args.max_cycles_iterations = iterations_per_launch_;
	args.wait_ns = wait_ns_;
	args.cta_row = cta_row_.get();
	args.cta_group = cta_group_.get();
	args.group_cta = group_cta_.get();
	args.agg_list = agg_list_.get();
	args.agg_list_offsets = agg_list_offsets_.get();
	args.cta_parts = tables_[0].get();
	args.part_start = tables_[1].get();
	args.part_nodes = tables_[2].get();
	args.part_offsets = tables_[3].get();
	args.part_list = tables_[4].get();
	args.group_agg = tables_[5].get();
	args.group_agg_offsets = tables_[6].get();
	args.coarse_part = coarse_part_.get();
	args.partial = partial_.get();
	args.R = R_.get();
	args.y = y_.get();
	args.tolerance_in = nullptr;
	args.tolerance_out = tolerance_.get();
	args.flags = flags_.get();
	args.status = reinterpret_cast<ResidentStatus*>(status_.get());
	args.barrier = &args.status->barrier;
	ResidentStatus total{};
	const auto copy = [&](double* to, const double* from) {
		CudaCheck(cudaMemcpyAsync(to, from, problem.entries()*sizeof(double), cudaMemcpyDeviceToDevice, stream),
			"resident GMRES start");
	};
	if (kind_ == kLeft2 || kind_ == kLeft2Fp32 || kind_ == kLeft4) {
		copy(problem.start, problem.x);
		total.kept = 1;
	}
	const auto give_up = [&]() {
		if (total.kept) copy(problem.x, problem.start);
		total.error = 4;
		fits_ = false;
		return total;
	};
	for (;;) {
		status_.Zero(stream);
		void* parameters[] = {&args};
		if (cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(KernelOf(kind_)), dim3(ctas_), dim3(threads_),
			parameters, smem_, stream) != cudaSuccess) {
			// fewer CTAs than planned can run together here, or no memory for the launch
			(void)cudaGetLastError();
			return give_up();
		}
		if (launches) *launches += 1;
		CudaCheck(cudaMemcpyAsync(host_, args.status, sizeof(ResidentStatus), cudaMemcpyDeviceToHost, stream),
			"resident GMRES status");
		CudaCheck(cudaStreamSynchronize(stream), "resident GMRES");
		total.converged = host_->converged;
		total.iterations += host_->iterations;
		total.error = host_->error;
		total.residual = host_->residual;
		total.kept |= host_->kept;
		if (total.error == 4) return give_up();
		if (total.error || total.converged || total.iterations >= problem.max_iterations || host_->iterations == 0)
			return total;
		args.tolerance_in = tolerance_.get();
		args.p.max_iterations = problem.max_iterations-total.iterations;
	}
}

} // namespace tfiga
