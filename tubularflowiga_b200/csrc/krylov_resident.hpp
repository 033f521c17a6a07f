// A whole (F)GMRES solve in one cooperative kernel (krylov_resident.cu), for systems whose Krylov
// basis fits the chip's shared memory.
#pragma once

#include "common.hpp"
#include "kernels.cuh"

#include <vector>

namespace tfiga {

// Device arrays of the two-level AMG that an application reads (Amg::ResidentView).
struct AmgResidentView {
	int coarse = 0;                          // aggregates; 0: no AMG
	const int32_t* agg = nullptr;            // aggregate of every fine node
	const double* mask = nullptr;            // [4 nodes] 1 = free
	const double* dense = nullptr;           // inverse of the coarse operator, rows dense_ld apart
	long long dense_ld = 0;
	double* coarse_x = nullptr;              // [4 coarse] scratch
	const int32_t* ap_rows = nullptr;        // A P: block rows of the fine nodes
	const int32_t* ap_cols = nullptr;
	const void* ap = nullptr;                // FP32 or FP64, as the matrix
	const double* inverse = nullptr;         // fine 4x4 block inverses
	double omega = 1.0;
	long long version = 0;                   // changes with the hierarchy
};

struct ResidentLowRank {
	int count = 0;
	const int* ptr = nullptr;
	const int* idx = nullptr;
	const double* val = nullptr;
	const double* coef = nullptr;
};

// What the kernel reports to the host.
struct ResidentStatus {
	int converged, iterations;
	int error;                               // 1 singular Hessenberg, 2 not finite, 4 a barrier wait ran out or no launch
	unsigned barrier;                        // arrivals at the grid barriers of this launch
	int kept;                                // 1 once x's start is kept in full
	double residual;
};

// One solve: pointers and scalars; the template arguments of the launch say which are used.
struct ResidentProblem {
	DevicePatternView pattern;
	const void* krylov_values = nullptr;     // operator of the Arnoldi products
	const void* residual_values = nullptr;   // operator of the true residual
	const double* rhs = nullptr;
	double* x = nullptr;
	double* start = nullptr;                 // scratch of x's size
	const double* inverse = nullptr;         // left block-Jacobi
	AmgResidentView amg;                     // right preconditioner of the flexible solve
	ResidentLowRank low;
	double* Z = nullptr;                     // flexible: [restart][n]
	void* V = nullptr;                       // basis: [restart + 1][n]
	double rtol = 0.0, tolerance_floor = 0.0;
	int max_iterations = 0;
	int fields = 4;
	std::size_t entries() const { return (std::size_t)fields*pattern.nodes; }
};

// Rows of every CTA, groups (independent segments) and work arrays of a matrix; laid out once.
class ResidentKrylov {
public:
	enum Kind { kLeft2, kLeft2Fp32, kLeft4, kFlexDouble, kFlexFloat, kFlexFloatFp64Basis, kKinds };
	~ResidentKrylov();
	// Whether a solve of this kind fits; lays out the plan when the kind, the hierarchy or the segments
	// (entry offsets, count + 1 values, or empty) are not those of the last call.
	bool Prepare(Kind kind, const DevicePatternView& pattern, int restart, const std::vector<int64_t>& segments,
		const AmgResidentView* amg, cudaStream_t stream);
	// Runs the solve and waits for it.  After a status with error 4 the plan is off (Prepare returns false) and x is as it
	// was before.
	ResidentStatus Solve(const ResidentProblem& problem, cudaStream_t stream, long long* launches);
	// Iterations after which a launch ends and the next one continues (checked between restart cycles), and the limit
	// of a wait at a grid barrier (0: any wait runs out).  Four seconds of wall clock: a barrier takes microseconds.
	// A plan that is off is made again.
	void SetLimits(int iterations_per_launch, long long wait_ns)
	{
		iterations_per_launch_ = iterations_per_launch;
		wait_ns_ = wait_ns;
		planned_ = false;
	}
private:
	void Plan(const DevicePatternView& pattern, const AmgResidentView* amg, cudaStream_t stream);
	void ReleaseArrays();
	bool planned_ = false, fits_ = false;
	Kind kind_ = kLeft4;
	std::vector<int64_t> segments_;
	long long amg_version_ = -1;
	int ctas_ = 0, groups_ = 1, restart_ = 0, slice_ = 0, pieces_ = 1, threads_ = 0;
	bool keep_ = false;
	int iterations_per_launch_ = 4096;
	long long wait_ns_ = 4000000000ll;
	size_t smem_ = 0;
	DeviceArray<int32_t> cta_row_, cta_group_, group_cta_, agg_list_, agg_list_offsets_;
	static constexpr int kTables = 7;
	DeviceArray<int32_t> tables_[kTables];   // restriction by CTA and group (see Args)
	DeviceArray<double> partial_, R_, y_, tolerance_, coarse_part_;
	DeviceArray<int> flags_;                 // group stop flags
	DeviceArray<int32_t> status_;            // a ResidentStatus
	ResidentStatus* host_ = nullptr;
};

} // namespace tfiga
