// Tensor-core (tcgen05) element tangent for the mixed-precision Newton path: the exact VMS tangent
// contracted with FP32 accumulation in tensor memory and added into an FP32 block-CSR Jacobian.
//
// Formulation: vms_tangent.cuh (NavierStokesElement.hpp:149-317 with the exact tangent :244-312).  Per row field i
// the tangent of an element is
//   K^{if}_{ab} = sum_k G^{if}[(b, f)][k] Psi[a][k],   k = (point, test feature): 64 x 4,
// with G from the points' numbers (LaunchPointStream, FP32) and the basis values.
//
// Organisation.  A CTA owns (element, row field): D is 256 rows (b, f) x up to 64 columns a, two
// M = 128 tiles in 128 columns of tensor memory.  What bounds it is making G, 64 x 1024 values per element and
// row field, on the CUDA cores; the products are small beside it.  So G never goes through shared memory: the
// thread that computes a row of G writes it to tensor memory (tcgen05.st), where the MMA takes its A operand from,
// and the factored form needs 8 to 13 multiply-adds per four values instead of 20.  Thread -> row: warp quarter
// q holds functions b = 32 (q & 1) + lane and column fields q >> 1 (tile 0) and 2 + (q >> 1) (tile 1), so both of
// a thread's columns share its basis values and L, column fields are warp-uniform (no divergence between the
// columns' different formulas), and a point's numbers are broadcast reads.  The two warps of a quarter take one of
// a chunk's two depth steps each; both points of a pair run in the halves of the packed FP32 operations.
// Chunks of eight points (two depth steps of K = 16: the waits and fences of a chunk cost a thread as much as a
// quarter of its arithmetic on four points).  Eight warps build; a ninth has one thread that issues the MMAs, a tenth
// (FP32 tables) one that fetches the chunks (bulk copies, three or four staged, across the items of a CTA: issuing them took the MMA thread
// 1,000 cycles a chunk).  They meet on mbarriers only (staged -> build -> unstaged, and full -> MMA -> empty; A and
// Psi, in shared memory with the 64-byte swizzle, are double-buffered): with a block barrier a chunk and one of the
// builders issuing, every chunk waited for that warp (37,000 cycles per CTA of which 12,000 waiting).  Waits are
// bounded in clock cycles.  Two CTAs per SM (256 tensor-memory columns each).
// Functions past the element's own are left out of N (steps of 16) and, from 32 down, of the second warp half.
// Epilogue: 16 columns a at a time through shared memory (a barrier a round where two rounds' worth fits), so that a thread has all
// four column fields of a block and adds 16 bytes at once (red.global.add.v4.f32).  Adding 8 bytes straight from the
// accumulators, without the barriers, is slower (tube below 6.09 ms against 5.80): the L2's additions per sector count.
// Cycles of an item (64 functions, two CTAs on the SM): build 11,000, Psi 2,500, epilogue 7,000, waits 6,500.
//
// Operands: BF16, split BF16 (hi + lo, three products) or TF32.
// Basis values come from the FP32 copy of the tables (coefficients / element organisation: one CTA per element and
// row field, or two persistent CTAs per SM) or, converted on the way, from the FP64 tables (fused organisation, which
// needs no copy).
//
// Measured, split BF16, against the kernel this replaces (G from 320 coefficients per point, through shared memory):
// 25,600-element tube 6.64 -> 5.57 ms, 3,264-element bifurcation 0.87 -> 0.69 ms; the coefficients it needed cost the
// point kernel 2.41 ms (now 1.05 ms) and 80 KiB per element (now 18).  From the FP64 tables 8.0 ms (before: 2.5 times
// the other organisation).
#include "common.hpp"
#include "kernels.cuh"
#include "vms_tangent.cuh"

#include <algorithm>
#include <cuda_bf16.h>

namespace tfiga {
namespace {

constexpr int kBuilders = 256;                   // building threads
// and a warp that issues the MMAs, and one that fetches; from the FP64 tables there is little to fetch (8.5 ms for the
// tube above with the warp, 8.0 without)
constexpr int Threads(bool fp64_tables) { return kBuilders+(fp64_tables ? 32 : 64); }
constexpr int kPoints = 8;                       // points per chunk: two depth steps of K = 16
constexpr int kChunks = kQuad/kPoints;
constexpr int kTmemCols = 256;                   // D: 2 x 64, A: 2 buffers x 2 depth steps x 2 tiles x 16
constexpr int kTmemA = 128;
constexpr long long kWaitCycles = 2000000000;   // about a second
constexpr int kEpilogueColumns = 16;

constexpr int kModeBf16 = 0, kModeSplit = 1, kModeTf32 = 2;

// Staged chunks, and epilogue rounds in shared memory: from the FP64 tables, which go through the L1, a slot and a round
// more cost more than they give (25,600-element tube 9.25 ms with four and two, 8.6 with three and one).
template <bool kFp64Tables> struct __align__(1024) TangentShared {
	static constexpr int kSlots = kFp64Tables ? 3 : 4, kRounds = kFp64Tables ? 1 : 2;
	unsigned char psi[2][2][64*64];              // B operand of a depth step: 64 rows a x 64 bytes, swizzled
	float2 phi[kSlots][kFeatures][kPoints/2][kMaxBasis];   // point pairs
	float2 pack[kSlots][kPoints/2][kPack];
	float out[kRounds][4][kEpilogueColumns][kMaxBasis];   // rounds of [column field][a][b]
	uint64_t staged[kSlots], unstaged[kSlots], full[2], empty[2];
	uint32_t tmem;
};
constexpr uint32_t kPhiBytes = kPoints/2*kMaxBasis*8;      // one feature of a chunk
constexpr uint32_t kPackBytes = kPoints/2*kPack*8;

// Instruction descriptor: D FP32, A and B BF16 (1) or TF32 (2), both K-major, M = 128.
__device__ __forceinline__ uint32_t InstructionDescriptor(bool tf32, int n)
{
	const uint32_t format = tf32 ? 2u : 1u;
	return (1u << 4) | (format << 7) | (format << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ uint32_t SmemAddress(const void* p)
{
	return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major, 64-byte swizzle: 8-row atoms of
// 512 B (stride byte offset 512), leading byte offset unused (1), version 1.
__device__ __forceinline__ uint64_t DescSw64(uint32_t address)
{
	return (uint64_t)((address >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46)
		| (4ull << 61);
}

// Byte offset of 16-byte chunk j (0..3) of row r in a 64-byte-swizzled K-major tile.
__device__ __forceinline__ int Sw64(int r, int j)
{
	return r*64+((j ^ ((r >> 1) & 3)) << 4);
}

__device__ __forceinline__ void MbarInit(uint64_t* bar, uint32_t count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(SmemAddress(bar)), "r"(count) : "memory");
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void MbarArrive(uint64_t* bar)
{
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(SmemAddress(bar)) : "memory");
}

__device__ __forceinline__ void MbarExpect(uint64_t* bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(SmemAddress(bar)), "r"(bytes)
		: "memory");
}

// Global -> shared bulk copy (16-byte aligned, a multiple of 16 bytes), counted on `bar`.
__device__ __forceinline__ void BulkCopy(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
		:: "r"(SmemAddress(dst)), "l"(src), "r"(bytes), "r"(SmemAddress(bar)) : "memory");
}

__device__ __forceinline__ bool MbarTryWait(uint32_t bar, uint32_t parity)
{
	uint32_t done;
	asm volatile("{\n\t.reg .pred p;\n\t"
		"mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
		"selp.u32 %0, 1, 0, p;\n\t}"
		: "=r"(done) : "r"(bar), "r"(parity) : "memory");
	return done != 0;
}

// Waits for completion of the mbarrier phase with the given parity, for at most kWaitCycles.
__device__ __noinline__ bool MbarWaitLonger(uint32_t bar, uint32_t parity)
{
	const long long start = clock64();
	while (!MbarTryWait(bar, parity))
		if (clock64()-start > kWaitCycles) return false;
	return true;
}
__device__ __forceinline__ bool MbarWaitBounded(uint64_t* bar, uint32_t parity)
{
	return MbarTryWait(SmemAddress(bar), parity) || MbarWaitLonger(SmemAddress(bar), parity);
}

// D (128 x N, FP32) (+)= A (128 x K, in tensor memory) B^T (N x K, in shared memory): K = 16 BF16 or 8 TF32.
// Nothing but A's address kind differs from the shared-memory form; A's lane is its row, and a 32-bit column
// holds two consecutive BF16 or one TF32.
__device__ __forceinline__ void MmaBf16(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\t"
		"setp.ne.b32 p, %4, 0;\n\t"
		"tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
		:: "r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}

__device__ __forceinline__ void MmaTf32(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\t"
		"setp.ne.b32 p, %4, 0;\n\t"
		"tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
		:: "r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}

__device__ __forceinline__ void MmaCommit(uint64_t* bar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
		:: "r"(SmemAddress(bar)) : "memory");
}

__device__ __forceinline__ void FenceBeforeSync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void FenceAfterSync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void FenceProxyAsync() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 lanes x 16 consecutive FP32 columns: thread l gets row (lane base + l), columns c .. c + 15.
__device__ __forceinline__ void TmemLoad16(uint32_t taddr, float v[16])
{
	uint32_t r[16];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
		"{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
		: "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
		  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
		: "r"(taddr));
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
	#pragma unroll
	for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// The calling warp's 32 lanes x 8 or 16 consecutive columns.
__device__ __forceinline__ void TmemStore8(uint32_t taddr, const uint32_t* r)
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
		:: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
		: "memory");
}
__device__ __forceinline__ void TmemStore16(uint32_t taddr, const uint32_t* r)
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
		"%14, %15, %16};"
		:: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
		"r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void TmemStoreWait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ uint32_t PackBf16(float lo, float hi)
{
	const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
	return *reinterpret_cast<const uint32_t*>(&v);
}

// x rounded to TF32 (10 fraction bits, nearest with ties away), as the 32-bit pattern the MMA reads.
__device__ __forceinline__ uint32_t Tf32(float x)
{
	uint32_t r;
	asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
	return r;
}

// Two FP32 values in one 64-bit register pair (first value in the low half), for the packed
// FP32 pipe of sm_100 (fma / sub .f32x2: one instruction for both halves).
__device__ __forceinline__ unsigned long long Pack2(float lo, float hi)
{
	unsigned long long d;
	asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
	return d;
}
__device__ __forceinline__ float Low(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float High(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ unsigned long long Fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
	unsigned long long d;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
	return d;
}
__device__ __forceinline__ unsigned long long Mul2(unsigned long long a, unsigned long long b)
{
	unsigned long long d;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
	return d;
}
__device__ __forceinline__ unsigned long long Sub2(unsigned long long a, unsigned long long b)
{
	unsigned long long d;
	asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
	return d;
}

// BF16 pair of a packed FP32 pair (low half -> low 16 bits).
__device__ __forceinline__ uint32_t Bf16Pair(unsigned long long v)
{
	return PackBf16(Low(v), High(v));
}

// The FP32 pair a BF16 pair stands for (exact).
__device__ __forceinline__ unsigned long long WidenBf16Pair(uint32_t h)
{
	return Pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u));
}

__device__ __forceinline__ void StoreShared16(uint32_t address, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
	asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(address), "r"(a), "r"(b), "r"(c), "r"(d)
		: "memory");
}

__device__ __forceinline__ void RedAdd4(float* p, float a, float b, float c, float d)
{
	asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" :: "l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
		: "memory");
}


// A packed pair of FP32 values (two points) for TangentColumn.
struct Pair {
	unsigned long long v;
};
__device__ __forceinline__ Pair Fma(Pair a, Pair b, Pair c) { return {Fma2(a.v, b.v, c.v)}; }
__device__ __forceinline__ Pair Mul(Pair a, Pair b) { return {Mul2(a.v, b.v)}; }

struct PairReader {
	const unsigned long long* p;
	__device__ __forceinline__ Pair operator()(int k) const { return {p[k]}; }
	__device__ __forceinline__ Two<Pair> two(int k) const
	{
		const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p+k);
		return {{v.x}, {v.y}};
	}
};

// Both of the thread's columns (fields kHalf and 2 + kHalf: tiles 0 and 1, sixteen columns apart) at the depth
// step's two point pairs, into its row of A.  Columns of a depth step: BF16 pairs of the points' hi parts, pair by
// pair and feature by feature, then the lo parts eight columns on; TF32: two columns per pair and feature.
template <int kMode, int I, int kHalf, class Shared>
__device__ __forceinline__ void BuildRows(const Shared& sm, int slot, int step, int b, Pair irho, Pair minus_nu,
	uint32_t column)
{
	uint32_t r[2][16];
	#pragma unroll
	for (int pair = 0; pair < 2; ++pair) {
		const PairReader pk{reinterpret_cast<const unsigned long long*>(&sm.pack[slot][2*step+pair][0])};
		const auto value = [&](int t) {
			return Pair{*reinterpret_cast<const unsigned long long*>(&sm.phi[slot][t][2*step+pair][b])};
		};
		const Pair n = value(0), g[3] = {value(1), value(2), value(3)};
		const Two<Pair> u01 = pk.two(kPackU);
		const Pair l = Fma(u01.a, g[0], Fma(u01.b, g[1], Fma(pk(kPackU+2), g[2], Mul(minus_nu, value(4)))));
		Pair v[2][4];
		TangentColumn<I, kHalf>(pk, n, g, l, irho, v[0]);
		TangentColumn<I, 2+kHalf>(pk, n, g, l, irho, v[1]);
		#pragma unroll
		for (int tile = 0; tile < 2; ++tile)
			#pragma unroll
			for (int s = 0; s < 4; ++s) {
				const unsigned long long x = v[tile][s].v;
				if constexpr (kMode == kModeTf32) {
					r[tile][8*pair+2*s] = Tf32(Low(x));
					r[tile][8*pair+2*s+1] = Tf32(High(x));
				} else {
					const uint32_t h = Bf16Pair(x);
					r[tile][4*pair+s] = h;
					r[tile][8+4*pair+s] = kMode == kModeSplit ? Bf16Pair(Sub2(x, WidenBf16Pair(h))) : 0u;
				}
			}
	}
	#pragma unroll
	for (int tile = 0; tile < 2; ++tile) {
		if constexpr (kMode == kModeBf16) TmemStore8(column+16*tile, r[tile]);
		else TmemStore16(column+16*tile, r[tile]);
	}
}

template <int kMode, bool kFp64Tables>
__global__ void __launch_bounds__(Threads(kFp64Tables), 2) TangentKernel(DeviceMeshView mesh, int items,
	const float* __restrict__ phi32, const double* __restrict__ phi64, const float* __restrict__ packs,
	const int32_t* __restrict__ element_blocks, float irho_value, float minus_nu_value, float* __restrict__ values,
	int* __restrict__ status)
{
	extern __shared__ unsigned char raw[];
	using Shared = TangentShared<kFp64Tables>;
	constexpr int kFetcher = kFp64Tables ? kBuilders : kBuilders+32;   // thread
	constexpr int kSlots = Shared::kSlots, kRounds = Shared::kRounds;
	Shared& sm = *reinterpret_cast<Shared*>(
		(reinterpret_cast<uintptr_t>(raw)+1023) & ~static_cast<uintptr_t>(1023));
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int quarter = warp & 3, group = warp >> 2;     // a quarter's two warps: depth steps, then tiles
	const auto functions = [&](int item) { return mesh.element_offsets[(item >> 2)+1]-mesh.element_offsets[item >> 2]; };
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
			:: "r"(SmemAddress(&sm.tmem)), "r"((uint32_t)kTmemCols) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	if (tid == 0) {
		for (int k = 0; k < kSlots; ++k) {
			MbarInit(&sm.staged[k], 1);
			MbarInit(&sm.unstaged[k], kBuilders/32);
		}
		for (int k = 0; k < 2; ++k) {
			MbarInit(&sm.full[k], kBuilders/32);
			MbarInit(&sm.empty[k], 1);
		}
	}
	FenceBeforeSync();
	__syncthreads();
	FenceAfterSync();
	const uint32_t tmem = sm.tmem;
	const Pair irho{Pack2(irho_value, irho_value)}, minus_nu{Pack2(minus_nu_value, minus_nu_value)};
	const int b = 32*(quarter & 1)+lane;
	bool failed = false;
	int ahead_nen = kFp64Tables ? 0 : functions(blockIdx.x);   // the next item's
	int first = 0;                               // chunks of the items before this one

	// Chunk number n of this CTA (counted over its items): slot n % kSlots, use n / kSlots of it; buffer n & 1, use
	// n / 2.  Chunks are fetched in this order across the items, so that an item's first ones arrive during the
	// epilogue before it.
	int fetched = 0;
	auto fetch = [&]() {
		const long long item = blockIdx.x+(long long)(fetched/kChunks)*gridDim.x;
		if (item >= items) return false;
		const int e = (int)(item >> 2), c = fetched%kChunks, slot = fetched%kSlots;
		MbarExpect(&sm.staged[slot], (kFp64Tables ? 0u : kFeatures*kPhiBytes)+kPackBytes);
		if constexpr (!kFp64Tables) {
			const float* P32 = phi32+(size_t)e*kFeatures*kQuad*kMaxBasis;
			#pragma unroll
			for (int t = 0; t < kFeatures; ++t)
				BulkCopy(&sm.phi[slot][t][0][0], P32+((size_t)t*(kQuad/2)+c*(kPoints/2))*kMaxBasis*2, kPhiBytes,
					&sm.staged[slot]);
		}
		BulkCopy(&sm.pack[slot][0][0], packs+(size_t)e*kQuad*kPack+(size_t)c*kPoints*kPack, kPackBytes, &sm.staged[slot]);
		++fetched;
		return true;
	};

	if constexpr (kFp64Tables)
		if (tid == kFetcher)
			for (int c = 0; c < kSlots; ++c) fetch();

	for (int item = blockIdx.x; item < items; item += gridDim.x, first += kChunks) {
		const int e = item >> 2, row = item & 3;
		int nen;
		if constexpr (kFp64Tables) {             // (no registers to spare)
			nen = functions(item);
		} else {
			nen = ahead_nen;
			if ((long long)item+gridDim.x < items) ahead_nen = functions(item+gridDim.x);
		}
		const int columns = (nen+15) & ~15;      // N of the product
		const auto wait = [&](uint64_t* bar, int use) {
			if (!failed) failed = !MbarWaitBounded(bar, (uint32_t)(use & 1));
		};
		if (warp == kBuilders/32) {
			if (lane == 0) {
				const uint32_t idesc = InstructionDescriptor(kMode == kModeTf32, columns);
				for (int c = 0; c < kChunks; ++c) {
					const int buffer = c & 1;
					wait(&sm.full[buffer], (first+c) >> 1);
					FenceAfterSync();
					#pragma unroll
					for (int step = 0; step < 2; ++step) {
						const uint64_t psi = DescSw64(SmemAddress(sm.psi[buffer][step]));
						const uint64_t psi_next = DescSw64(SmemAddress(sm.psi[buffer][step])+32);
						const uint32_t accumulate = c > 0 || step > 0 ? 1u : 0u;
						const uint32_t a = tmem+kTmemA+64*buffer+32*step;
						// the tiles in turn: consecutive products accumulate into different columns
						const auto both = [&](uint32_t offset, uint64_t operand, uint32_t add) {
							#pragma unroll
							for (int tile = 0; tile < 2; ++tile)
								if constexpr (kMode == kModeTf32) MmaTf32(tmem+64*tile, a+16*tile+offset, operand, idesc, add);
								else MmaBf16(tmem+64*tile, a+16*tile+offset, operand, idesc, add);
						};
						both(0, psi, accumulate);                              // hi hi; TF32: the first eight k
						if constexpr (kMode == kModeSplit) {
							both(0, psi_next, 1u);                             // hi lo
							both(8, psi, 1u);                                  // lo hi
						}
						if constexpr (kMode == kModeTf32) both(8, psi_next, 1u);
					}
					MmaCommit(&sm.empty[buffer]);
					// every builder is done with chunk c's slot
					if constexpr (kFp64Tables) if (!failed) fetch();
				}
			}
			__syncwarp();
		} else if (warp > kBuilders/32) {
			// up to kSlots chunks ahead of the builders, into the next item
			if (lane == 0)
				while (fetched < first+kChunks+kSlots && !failed) {
					if (fetched >= kSlots) wait(&sm.unstaged[fetched%kSlots], fetched/kSlots-1);
					if (failed || !fetch()) break;
				}
			__syncwarp();
		} else {
		const double* P64 = kFp64Tables ? phi64+(size_t)e*kFeatures*kQuad*kMaxBasis : nullptr;
		float held[2][kFeatures];                // FP64 tables: points tid / 64 and 4 + tid / 64, function tid % 64
		auto load_fp64 = [&](int c) {
			const int a = tid & 63;
			#pragma unroll
			for (int h = 0; h < 2; ++h)
				#pragma unroll
				for (int t = 0; t < kFeatures; ++t)
					held[h][t] = a < columns
						? (float)__ldg(P64+((size_t)t*kQuad+c*kPoints+4*h+(tid >> 6))*kMaxBasis+a) : 0.0f;
		};
		auto store_fp64 = [&](int slot) {
			const int a = tid & 63;
			#pragma unroll
			for (int h = 0; h < 2; ++h) {
				const int q = 4*h+(tid >> 6);
				#pragma unroll
				for (int t = 0; t < kFeatures; ++t)
					reinterpret_cast<float*>(&sm.phi[slot][t][q >> 1][a])[q & 1] = held[h][t];
			}
		};
		const auto builders_sync = [] { asm volatile("bar.sync 1, %0;" :: "n"(kBuilders) : "memory"); };
		if constexpr (kFp64Tables) load_fp64(0);
		for (int c = 0; c < kChunks; ++c) {
			const int n = first+c, slot = n%kSlots, buffer = c & 1;
			if constexpr (kFp64Tables) {
				// (the slot's readers of three chunks ago have passed two of these barriers since)
				store_fp64(slot);
				if (c+1 < kChunks) load_fp64(c+1);
				builders_sync();
			}
			wait(&sm.staged[slot], n/kSlots);
			if (n >= 2) wait(&sm.empty[buffer], (n >> 1)-1);   // the MMAs that read these buffers last
			FenceAfterSync();
			// A: this thread's rows
			if (32*(quarter & 1) < nen) {
				const uint32_t column = tmem+((uint32_t)(32*quarter) << 16)+kTmemA+64*buffer+32*group;
				switch (2*row+(quarter >> 1)) {
				case 0: BuildRows<kMode, 0, 0>(sm, slot, group, b, irho, minus_nu, column); break;
				case 1: BuildRows<kMode, 0, 1>(sm, slot, group, b, irho, minus_nu, column); break;
				case 2: BuildRows<kMode, 1, 0>(sm, slot, group, b, irho, minus_nu, column); break;
				case 3: BuildRows<kMode, 1, 1>(sm, slot, group, b, irho, minus_nu, column); break;
				case 4: BuildRows<kMode, 2, 0>(sm, slot, group, b, irho, minus_nu, column); break;
				case 5: BuildRows<kMode, 2, 1>(sm, slot, group, b, irho, minus_nu, column); break;
				case 6: BuildRows<kMode, 3, 0>(sm, slot, group, b, irho, minus_nu, column); break;
				default: BuildRows<kMode, 3, 1>(sm, slot, group, b, irho, minus_nu, column); break;
				}
			}
			// Psi: row a, two test features of one point pair per depth step (k = 8 pair + 2 feature + point of the
			// pair: a thread's values are 16-byte units hi and lo of its row)
			{
				const int a = tid & 63, step = tid >> 7, pair = (tid >> 6) & 1;
				if (a < columns) {
					const uint32_t base = SmemAddress(sm.psi[buffer][step]);
					uint32_t h[4], o[4];
					unsigned long long v[4];
					#pragma unroll
					for (int s = 0; s < 4; ++s)
						v[s] = *reinterpret_cast<const unsigned long long*>(&sm.phi[slot][s][2*step+pair][a]);
					if constexpr (kMode == kModeTf32) {
						StoreShared16(base+Sw64(a, 2*pair), Tf32(Low(v[0])), Tf32(High(v[0])), Tf32(Low(v[1])),
							Tf32(High(v[1])));
						StoreShared16(base+Sw64(a, 2*pair+1), Tf32(Low(v[2])), Tf32(High(v[2])), Tf32(Low(v[3])),
							Tf32(High(v[3])));
					} else {
						#pragma unroll
						for (int s = 0; s < 4; ++s) h[s] = Bf16Pair(v[s]);
						StoreShared16(base+Sw64(a, pair), h[0], h[1], h[2], h[3]);
						if constexpr (kMode == kModeSplit) {
							#pragma unroll
							for (int s = 0; s < 4; ++s) o[s] = Bf16Pair(Sub2(v[s], WidenBf16Pair(h[s])));
							StoreShared16(base+Sw64(a, 2+pair), o[0], o[1], o[2], o[3]);
						}
					}
				}
			}
			TmemStoreWait();
			FenceBeforeSync();
			FenceProxyAsync();
			__syncwarp();
			if (lane == 0) {
				MbarArrive(&sm.full[buffer]);
				if constexpr (!kFp64Tables) MbarArrive(&sm.unstaged[slot]);
			}
		}

		// warp (tile, quarter): column field 2 tile + (quarter >> 1) of functions b for sixteen a at a time
		const int field = 2*group+(quarter >> 1);
		const int32_t* EB = element_blocks+(size_t)e*kMaxBasis*kMaxBasis;
		float* base = values+4*row;
		const int ob = tid & 63, oa = tid >> 6;
		auto blocks_of = [&](int a0, int block[4]) {
			#pragma unroll
			for (int k = 0; k < 4; ++k) {
				const int a = a0+oa+4*k;
				block[k] = a < nen && ob < nen ? __ldg(EB+a*kMaxBasis+ob) : -1;
			}
		};
		int block[4];
		blocks_of(0, block);
		// the last commits of both buffers, before the accumulators are read
		wait(&sm.empty[0], ((first+kChunks) >> 1)-1);
		wait(&sm.empty[1], ((first+kChunks) >> 1)-1);
		FenceAfterSync();
		for (int a0 = 0; a0 < columns; a0 += kEpilogueColumns) {
			const int round = a0/kEpilogueColumns%kRounds;   // (two: its last readers have passed a barrier since)
			if (32*(quarter & 1) < nen) {
				float v[16];
				TmemLoad16(tmem+((uint32_t)(32*quarter) << 16)+64*group+a0, v);
				#pragma unroll
				for (int k = 0; k < 16; ++k) sm.out[round][field][k][b] = v[k];
			}
			int ahead[4] = {-1, -1, -1, -1};
			if (a0+kEpilogueColumns < columns) blocks_of(a0+kEpilogueColumns, ahead);
			builders_sync();
			#pragma unroll
			for (int k = 0; k < 4; ++k)
				if (block[k] >= 0)
					RedAdd4(base+(size_t)block[k]*16, sm.out[round][0][oa+4*k][ob], sm.out[round][1][oa+4*k][ob],
						sm.out[round][2][oa+4*k][ob], sm.out[round][3][oa+4*k][ob]);
			if constexpr (kRounds == 1) builders_sync();
			#pragma unroll
			for (int k = 0; k < 4; ++k) block[k] = ahead[k];
		}
		}
		// the accumulators are free for the next item, and a failed wait ends the CTA
		FenceBeforeSync();
		if (__syncthreads_or(failed)) { failed = true; break; }
		FenceAfterSync();
	}
	if (failed && tid == kFetcher)               // copies in flight land before the CTA ends
		for (int n = max(0, fetched-kSlots); n < fetched; ++n) MbarWaitBounded(&sm.staged[n%kSlots], n/kSlots & 1);
	__syncthreads();
	if (failed && tid == 0) atomicOr(status, 1);
	if (warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"((uint32_t)kTmemCols));
}

// Loads the kernel and allows its shared memory (bytes returned).
template <int kMode, bool kFp64Tables>
int Configure()
{
	const int bytes = (int)sizeof(TangentShared<kFp64Tables>)+1024;
	CudaCheck(cudaFuncSetAttribute(TangentKernel<kMode, kFp64Tables>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		bytes), "tangent shared memory");
	return bytes;
}

template <int kMode, bool kFp64Tables>
void Launch(const DeviceMeshView& mesh, const float* phi32, const double* phi64, const float* packs,
	const int32_t* element_blocks, AssemblyParams params, float* values, int* status, bool persistent,
	cudaStream_t stream)
{
	const long long items = 4LL*mesh.elements;
	if (items == 0) return;
	if (items > 0x7fffffffLL) Fail(-7, "too many elements for one tangent launch");
	const int bytes = Configure<kMode, kFp64Tables>();
	long long grid = items;
	if (persistent) {
		int device = 0, sms = 0;
		CudaCheck(cudaGetDevice(&device), "device");
		CudaCheck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "device attribute");
		grid = std::min<long long>(items, 2LL*sms);
	}
	TangentKernel<kMode, kFp64Tables><<<(unsigned)grid, Threads(kFp64Tables), bytes, stream>>>(mesh, (int)items, phi32, phi64,
		packs, element_blocks, (float)(1.0/params.density), (float)(-params.viscosity/params.density), values, status);
	LaunchCheck("TangentKernel");
}

template <bool kFp64Tables>
void LaunchMode(const DeviceMeshView& mesh, const float* phi32, const double* phi64, const float* packs,
	const int32_t* element_blocks, AssemblyParams params, float* values, int* status, int operands, bool persistent,
	cudaStream_t stream)
{
	if (operands == TC_OPERANDS_SPLIT)
		Launch<kModeSplit, kFp64Tables>(mesh, phi32, phi64, packs, element_blocks, params, values, status, persistent,
			stream);
	else if (operands == TC_OPERANDS_TF32)
		Launch<kModeTf32, kFp64Tables>(mesh, phi32, phi64, packs, element_blocks, params, values, status, persistent,
			stream);
	else
		Launch<kModeBf16, kFp64Tables>(mesh, phi32, phi64, packs, element_blocks, params, values, status, persistent,
			stream);
}

} // namespace

void LoadTangentTc(int operands)
{
	if (operands == TC_OPERANDS_SPLIT) Configure<kModeSplit, false>(), Configure<kModeSplit, true>();
	else if (operands == TC_OPERANDS_TF32) Configure<kModeTf32, false>(), Configure<kModeTf32, true>();
	else Configure<kModeBf16, false>(), Configure<kModeBf16, true>();
}

void LaunchTangentTc(const DeviceMeshView& mesh, int first, int count, const float* phi32, const double* phi,
	const float* packs, const int32_t* element_blocks, AssemblyParams params, float* values, int* status, int operands,
	bool persistent, cudaStream_t stream)
{
	// the arrays by element begin at `first`
	DeviceMeshView view = mesh;
	view.elements = count;
	view.element_offsets += first;
	element_blocks += (size_t)first*kMaxBasis*kMaxBasis;
	const size_t tables = (size_t)first*kFeatures*kQuad*kMaxBasis;
	if (phi32)
		LaunchMode<false>(view, phi32+tables, nullptr, packs, element_blocks, params, values, status, operands, persistent,
			stream);
	else
		LaunchMode<true>(view, nullptr, phi+tables, packs, element_blocks, params, values, status, operands, persistent,
			stream);
}

} // namespace tfiga
