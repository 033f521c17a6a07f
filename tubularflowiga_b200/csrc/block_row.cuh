// One 4x4 block row of A x.
//
// Four lanes share a block, one row of it each, so that a warp reads eight consecutive blocks at once, contiguously
// (16 bytes per lane of FP32 values, two times 16 of FP64), and a row's sum needs three shuffles.  Several such
// groups are in flight per warp.  With a whole block per lane the 16-byte loads of a warp lay 64 or 128 bytes apart:
// FP64 products ran at 3.6 TB/s (2.4 GB matrix of 58,145 rows: 383 us, now 224), FP32 ones of matrices near the L2's
// size at 4.8 TB/s (207 MB: 43 us, now 39).  kParts warps share a row where a warp per row would leave the chip's
// schedulers idle; kStream: values are loaded to leave the L2 first (a matrix that does not fit it).
#pragma once

#include "kernels.cuh"

namespace tfiga {

template <bool kStream, class V> __device__ __forceinline__ V LoadMatrix(const V* p)
{
	if constexpr (kStream) return __ldcs(p);
	else return __ldg(p);
}

// Row r of a 4x4 block, and its product with the block column's four vector entries added to s.
template <class T> struct BlockRow;
template <> struct BlockRow<float> {
	float4 q;
	template <bool kStream> __device__ __forceinline__ void Load(const float* v, size_t block, int r)
	{
		q = LoadMatrix<kStream>(reinterpret_cast<const float4*>(v+block*16+4*r));
	}
	__device__ __forceinline__ double Dot(double2 x, double2 y, double s) const
	{
		s = fma((double)q.x, x.x, s); s = fma((double)q.y, x.y, s);
		return fma((double)q.w, y.y, fma((double)q.z, y.x, s));
	}
};
template <> struct BlockRow<double> {
	double2 a, b;
	template <bool kStream> __device__ __forceinline__ void Load(const double* v, size_t block, int r)
	{
		const double2* q = reinterpret_cast<const double2*>(v+block*16+4*r);
		a = LoadMatrix<kStream>(q);
		b = LoadMatrix<kStream>(q+1);
	}
	__device__ __forceinline__ double Dot(double2 x, double2 y, double s) const
	{
		s = fma(a.x, x.x, s); s = fma(a.y, x.y, s);
		return fma(b.y, y.y, fma(b.x, y.x, s));
	}
};

// The sum of row r = lane & 3 over the warp's eight block groups.
__device__ __forceinline__ double QuadRowSum(double s)
{
	#pragma unroll
	for (int o = 16; o >= 4; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	return s;
}

// Part `part` of kParts of (A x)[4*row + r], in lanes with lane & 3 == r.  kPairs: a row's remainder by twos.
template <class T, int kParts, bool kStream, bool kPairs>
__device__ __forceinline__ double RowBlockDot(const DevicePatternView& p, const T* __restrict__ values,
	const double* __restrict__ x, int row, int part, int lane)
{
	// groups of eight blocks in flight: as many as registers and a part's length allow
	constexpr int kUnroll = sizeof(T) == 4 ? 4 : kParts == 4 ? 2 : kParts == 1 && kStream ? 8 : 4;
	const int b0 = p.row_offsets[row], b1 = p.row_offsets[row+1];
	const int per = (b1-b0+kParts-1)/kParts;
	const int lo = min(b1, b0+part*per), hi = min(b1, lo+per);
	const int r = lane & 3;
	double s = 0.0;
	int b = lo+(lane >> 2);
	for (; b+8*(kUnroll-1) < hi; b += 8*kUnroll) {
		int c[kUnroll];
		BlockRow<T> a[kUnroll];
		#pragma unroll
		for (int u = 0; u < kUnroll; ++u) c[u] = __ldg(p.columns+b+8*u);
		#pragma unroll
		for (int u = 0; u < kUnroll; ++u) a[u].template Load<kStream>(values, (size_t)(b+8*u), r);
		#pragma unroll
		for (int u = 0; u < kUnroll; ++u) {
			const double2* v = reinterpret_cast<const double2*>(x+4*(size_t)c[u]);
			s = a[u].Dot(__ldg(v), __ldg(v+1), s);
		}
	}
	if constexpr (kPairs) {
		// what is left by twos, in predicated loads: half the round trips to memory of the loop below
		#pragma unroll 1
		for (; b-(lane >> 2) < hi; b += 16) {
			int c[2];
			BlockRow<T> a[2];
			#pragma unroll
			for (int u = 0; u < 2; ++u) c[u] = b+8*u < hi ? __ldg(p.columns+b+8*u) : -1;
			#pragma unroll
			for (int u = 0; u < 2; ++u)
				if (c[u] >= 0) a[u].template Load<kStream>(values, (size_t)(b+8*u), r);
			#pragma unroll
			for (int u = 0; u < 2; ++u)
				if (c[u] >= 0) {
					const double2* v = reinterpret_cast<const double2*>(x+4*(size_t)c[u]);
					s = a[u].Dot(__ldg(v), __ldg(v+1), s);
				}
		}
	} else {
		for (; b < hi; b += 8) {
			const double2* v = reinterpret_cast<const double2*>(x+4*(size_t)__ldg(p.columns+b));
			BlockRow<T> a;
			a.template Load<kStream>(values, (size_t)b, r);
			s = a.Dot(__ldg(v), __ldg(v+1), s);
		}
	}
	return QuadRowSum(s);
}

} // namespace tfiga
