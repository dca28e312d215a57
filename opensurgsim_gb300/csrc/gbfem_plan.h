// gbfem_plan.h -- host-side plans of the resident CG (gbfem_res.cu): which CTA holds which rows.
#pragma once

#include <vector>

#include "gbfem_res.h"

namespace gbfem {

// One way to spread the systems of a handle over CTAs.
struct ResPlan
{
	bool ok = false;
	int form = 0;                 // ResForm whose layout the shares were sized for
	int grid = 0;                 // CTAs of a launch
	std::vector<ResPart> parts;   // by system, then by place in the system
	std::vector<int> segPart;     // systems + 1: first part of each
	std::vector<int> halo;
	std::vector<uint16_t> lcol;
	std::vector<int> chunkWarp, chunkList;  // mixed forms
	size_t mailWords = 0;
	std::vector<int2> tasks;      // every share once, longest systems first
};

// Position of each of n points (3 coordinates each) along a Morton curve through cells of about two points'
// spacing: the order in which 32 consecutive rows of a system are close together.
std::vector<uint32_t> res_curve_keys(const double* points, int n);

// Order of a system's SELL chunks in which contiguous ranges are compact: recursive bisection of the
// chunk centroids (3 per chunk) at half the weight along the longest side.
std::vector<int> res_chunk_order(const std::vector<double>& centroid, const std::vector<int>& weight);

// Parts of a system's nodes (indices 0..n-1 into points and weight) for `g` shares: compact boxes of about
// equal weight, every part but the last a multiple of 32 nodes.
std::vector<std::vector<int>> res_node_parts(const double* points, const std::vector<int>& weight, int g);

// Cut of the chunks [first, last) in their order into g ranges of about equal weight: g + 1 bounds.
std::vector<int> res_cut(const std::vector<int>& off, int first, int last, int g);

// Weight of a chunk of `slots` SELL slots in a share: its slots and its rows' own work.
inline int res_chunk_weight(int slots) { return slots + 4; }

// Shares (CTAs) each system gets of `ctas` resident ones. segWeight / segChunks: total chunk weight and chunks of each.
// local: expected local rows (own and halo) an own row; cost: expected iterations of each, up to a factor.
std::vector<int> res_widths(int form, double local, const std::vector<long long>& segWeight,
							const std::vector<int>& segChunks, const std::vector<double>& cost, int ctas, int smemBudget);

// Plan of the systems whose shares are the chunk ranges between consecutive bounds cut[s], on the SELL
// matrix (off, rcol: columns as row positions), for `ctas` resident CTAs; cost[s] > 0: expected iterations, which
// only orders the systems. ok is false when a share's vectors do not fit in smemBudget bytes.
ResPlan res_plan(int form, const std::vector<std::vector<int>>& cut, const std::vector<int>& off,
				 const std::vector<int>& rcol, const std::vector<double>& cost, int ctas, int smemBudget);

// Whether the plan's shares fit another form's layout.
bool res_fits(const ResPlan& plan, int form, int smemBudget);

// Dynamic shared memory of a launch: the largest share with its whole matrix, at most the budget.
size_t res_smem(const ResPlan& plan, int form, const std::vector<int>& off, int smemBudget);

}  // namespace gbfem
