// gbfem_plan.cpp -- host-side plans of the resident CG (gbfem_res.cu).

#include "gbfem_plan.h"

#include <algorithm>
#include <cmath>
#include <limits>
#include <numeric>
#include <utility>

namespace gbfem {
namespace {

// Sorts indices by every third value from `coordinate`, then by index; the keys sit beside them for the sort. A node of no
// element may lie anywhere, also at NaN, which has no place in an order: such nodes come last.
void sort_along(const double* coordinate, int* first, int* last)
{
	std::vector<std::pair<double, int>> key(last - first);
	for (int* i = first; i != last; ++i)
	{
		const double v = coordinate[3 * (size_t)*i];
		key[i - first] = {std::isnan(v) ? std::numeric_limits<double>::infinity() : v, *i};
	}
	std::sort(key.begin(), key.end());
	for (int* i = first; i != last; ++i) *i = key[i - first].second;
}

void bisect(const std::vector<double>& c, const std::vector<int>& w, int* first, int* last)
{
	const int n = (int)(last - first);
	if (n <= 1) return;
	double lo[3], hi[3];
	for (int k = 0; k < 3; ++k) lo[k] = hi[k] = c[3 * (size_t)first[0] + k];
	for (int i = 1; i < n; ++i)
		for (int k = 0; k < 3; ++k)
		{
			lo[k] = std::min(lo[k], c[3 * (size_t)first[i] + k]);
			hi[k] = std::max(hi[k], c[3 * (size_t)first[i] + k]);
		}
	int axis = 0;
	for (int k = 1; k < 3; ++k)
		if (hi[k] - lo[k] > hi[axis] - lo[axis]) axis = k;
	sort_along(c.data() + axis, first, last);
	long long total = 0, run = 0;
	for (int i = 0; i < n; ++i) total += w[first[i]];
	int cut = 0;
	while (cut < n - 1 && 2 * (run + w[first[cut]]) <= total) run += w[first[cut++]];
	cut = std::max(1, cut);
	bisect(c, w, first, first + cut);
	bisect(c, w, first + cut, last);
}

// Cuts nodes[first, last) (whose number is a multiple of 32, or which end the system) into g parts.
void split_nodes(const double* X, const std::vector<int>& w, int* first, int* last, int g, std::vector<std::vector<int>>& out)
{
	const int n = (int)(last - first);
	if (g == 1)
	{
		out.emplace_back(first, last);
		return;
	}
	double lo[3], hi[3];
	for (int k = 0; k < 3; ++k) lo[k] = hi[k] = X[3 * (size_t)first[0] + k];
	for (int i = 1; i < n; ++i)
		for (int k = 0; k < 3; ++k)
		{
			lo[k] = std::min(lo[k], X[3 * (size_t)first[i] + k]);
			hi[k] = std::max(hi[k], X[3 * (size_t)first[i] + k]);
		}
	int axis = 0;
	for (int k = 1; k < 3; ++k)
		if (hi[k] - lo[k] > hi[axis] - lo[axis]) axis = k;
	sort_along(X + axis, first, last);
	long long total = 0, run = 0;
	for (int i = 0; i < n; ++i) total += w[first[i]];
	const int gl = g / 2;
	int cut = 0;
	while (cut < n && run * g < total * gl) run += w[first[cut++]];
	cut = (cut + 16) / 32 * 32;
	cut = std::min(std::max(cut, 32 * gl), (n + 31) / 32 * 32 - 32 * (g - gl));
	split_nodes(X, w, first, first + cut, gl, out);
	split_nodes(X, w, first + cut, last, g - gl, out);
}

}  // namespace

std::vector<std::vector<int>> res_node_parts(const double* points, const std::vector<int>& weight, int g)
{
	std::vector<int> nodes(weight.size());
	std::iota(nodes.begin(), nodes.end(), 0);
	std::vector<std::vector<int>> parts;
	split_nodes(points, weight, nodes.data(), nodes.data() + nodes.size(), g, parts);
	return parts;
}

std::vector<int> res_cut(const std::vector<int>& off, int first, int last, int g)
{
	std::vector<int> cut(1, first);
	long long total = 0, run = 0;
	for (int c = first; c < last; ++c) total += res_chunk_weight(off[c + 1] - off[c]);
	int c = first;
	for (int r = 0; r + 1 < g; ++r)
	{
		// Up to the chunk whose middle passes this range's end, leaving a chunk for each range after it.
		while (c < last - (g - 1 - r))
		{
			const int w = res_chunk_weight(off[c + 1] - off[c]);
			if (c > cut.back() && (2 * run + w) * g > 2 * total * (r + 1)) break;
			run += w;
			++c;
		}
		cut.push_back(c);
	}
	cut.push_back(last);
	return cut;
}

std::vector<uint32_t> res_curve_keys(const double* points, int n)
{
	std::vector<uint32_t> key(n, 0);
	double lo[3], hi[3], volume = 1.0;
	for (int k = 0; k < 3; ++k) lo[k] = hi[k] = n ? points[k] : 0.0;
	for (int i = 0; i < n; ++i)
		for (int k = 0; k < 3; ++k)
		{
			lo[k] = std::min(lo[k], points[3 * (size_t)i + k]);
			hi[k] = std::max(hi[k], points[3 * (size_t)i + k]);
		}
	int dims = 0;
	for (int k = 0; k < 3; ++k)
		if (hi[k] > lo[k])
		{
			volume *= hi[k] - lo[k];
			++dims;
		}
	if (dims == 0) return key;
	double cell = 2.0 * std::pow(volume / n, 1.0 / dims);
	for (int k = 0; k < 3; ++k) cell = std::max(cell, (hi[k] - lo[k]) / 1023.0);
	if (!(cell > 0.0) || !std::isfinite(cell)) return key;
	for (int i = 0; i < n; ++i)
		for (int k = 0; k < 3; ++k)
		{
			const uint32_t q = (uint32_t)std::min(1023.0, (points[3 * (size_t)i + k] - lo[k]) / cell);
			for (int b = 0; b < 10; ++b) key[i] |= ((q >> b) & 1u) << (3 * b + k);
		}
	return key;
}

std::vector<int> res_chunk_order(const std::vector<double>& centroid, const std::vector<int>& weight)
{
	std::vector<int> order(weight.size());
	std::iota(order.begin(), order.end(), 0);
	if (!order.empty()) bisect(centroid, weight, order.data(), order.data() + order.size());
	return order;
}

std::vector<int> res_widths(int form, double local, const std::vector<long long>& segWeight,
							const std::vector<int>& segChunks, const std::vector<double>& cost, int ctas, int smemBudget)
{
	const int nseg = (int)segWeight.size();
	// Bytes of a row's vectors, its own and its part of the halo, and of a slot. A share takes up to `scale`
	// times the shared memory: what does not fit is read from L2 in every product, which costs less than the
	// waits of more and smaller shares (64 meshes, mixed: 7.0 ms a solve at 2, 5.7 at 2.5, 6.0 at 3, 6.6 at 3.5;
	// 24 meshes, FP64: 3.9 ms at 1, 3.3 at 1.5, 3.7 at 2).
	const double scale = res_mixed(form) ? 2.5 : 1.5;
	const int vecs = (int)(local * res_loc_bytes(form)) + res_own_bytes(form) + 4;
	const int slot = res_layout(form, 1, 0).slotBytes;
	const double room = smemBudget - (kResPieces * 32.0 * res_part_bytes(form) + 2048.0);
	// Where CTAs are left over, shares shrink to this weight: below it an iteration is all exchange (mixed, 1,331
	// nodes: 0.254 ms a solve at 40, 0.265 at 50, 0.279 at 80, 0.304 at 120; whole steps in a graph at 40, 45, 50 and 60:
	// 216 nodes 239, 239, 242, 242 us, 512 252, 252, 254, 273, 1,331 257, 263, 273, 273, 2,744 310, 298, 298, 298,
	// 4,913 325, 328, 328, 335;
	// FP64 1,331 nodes: 0.58 ms at 14, 0.65 at 20, 0.82 at 50; 17,280 scalar rows: 0.54 ms at 126, 0.50 at 250,
	// 0.56 at 400). Past 128 CTAs the sums take a third poll (18,081 nodes: 0.415 ms on 128, 0.443 on 152; FP64
	// 29,184 nodes 1.19 and 1.23).
	const double least = res_mixed(form) ? 45.0 : (form == kResF64S ? 200.0 : 14.0);
	std::vector<int> width(nseg), most(nseg);
	long long total = 0;
	for (int s = 0; s < nseg; ++s)
	{
		const double rows = segChunks[s] * 32.0, matrix = (double)(segWeight[s] - 4LL * segChunks[s]) * slot;
		const double need = std::max(rows * vecs / 0.95, (rows * vecs + matrix) / scale) / room;
		total += width[s] = std::max(1, std::min((int)(need * 1.02 + 1.0), std::min(ctas, segChunks[s])));
	}
	for (int s = 0; s < nseg; ++s)
		most[s] = std::max(width[s], std::min({ctas, 128, segChunks[s], (int)(segWeight[s] / least)}));
	if (nseg == 1)
	{
		// One cluster rather than a few CTAs more: its exchanges are shorter (mixed 1,728 nodes 0.232 ms a solve on
		// 16 CTAs, 0.258 on 20; 2,744 0.266 and 0.270 on 32; 3,024 0.281 and 0.274 on 35; FP64 576 nodes 0.404 on 16
		// and 0.473 on 18, 729 0.497 and 0.473 on 23).
		const int need = width[0];
		width[0] = most[0];
		if (need <= kResCluster && width[0] > kResCluster && width[0] <= (res_mixed(form) ? 32 : 20)) width[0] = kResCluster;
	}
	else
	{
		// The CTAs left over go one by one to the system expected to end last: its iterations times an
		// iteration's waits and its share's work (all systems widened alike: 36 FP64 meshes of 300 to 2,100 cubes
		// 2.55 ms a solve, here 2.02; 16 of 800 to 4,000 2.54 and 2.14; 20 mixed ones of 500 to 12,500 1.21 and
		// 0.92). Systems that take more CTAs than there are go in turn, the longest first: squeezing them into one
		// turn was slower (24 FP64 meshes of 500 to 8,000 cubes 3.65 ms, in turn 3.01).
		const double wait = res_mixed(form) ? 2.7 : 6.5, work = res_mixed(form) ? 0.012 : 0.07;
		auto time = [&](int s) { return cost[s] * (wait + work * segWeight[s] / width[s]); };
		auto later = [&](int a, int b) { return time(a) < time(b); };
		std::vector<int> heap;
		for (int s = 0; s < nseg; ++s)
			if (width[s] < most[s]) heap.push_back(s);
		std::make_heap(heap.begin(), heap.end(), later);
		for (; total < ctas && !heap.empty(); ++total)
		{
			std::pop_heap(heap.begin(), heap.end(), later);
			const int s = heap.back();
			if (++width[s] < most[s])
				std::push_heap(heap.begin(), heap.end(), later);
			else
				heap.pop_back();
		}
	}
	for (int& w : width) w = std::min(w, kResMaxGroup);
	return width;
}

ResPlan res_plan(int form, const std::vector<std::vector<int>>& cut, const std::vector<int>& off,
				 const std::vector<int>& rcol, const std::vector<double>& cost, int ctas, int smemBudget)
{
	ResPlan plan;
	plan.form = form;
	const int nseg = (int)cut.size();
	const int nrows = 32 * cut.back().back();
	plan.segPart.assign(1, 0);
	plan.lcol.assign(rcol.size(), 0);
	std::vector<int> local(nrows, -1);  // local index of a halo row in the current share
	std::vector<int> width(nseg);
	for (int s = 0; s < nseg; ++s)
	{
		const int g = width[s] = (int)cut[s].size() - 1;
		if (g < 1 || g > kResMaxGroup || g > ctas) return plan;
		for (int r = 0; r < g; ++r)
		{
			ResPart p{};
			p.seg = s;
			p.rank = r;
			p.g = g;
			p.c0 = cut[s][r];
			p.c1 = cut[s][r + 1];
			if (p.c1 <= p.c0) return plan;
			p.mail0 = (int)plan.mailWords;
			p.h0 = (int)plan.halo.size();
			const int r0 = 32 * p.c0, r1 = 32 * p.c1;
			for (size_t k = 32 * (size_t)off[p.c0]; k < 32 * (size_t)off[p.c1]; ++k)
			{
				const int J = rcol[k];
				if (J < r0 || J >= r1)
				{
					if (local[J] < 0)
					{
						local[J] = r1 - r0 + (int)plan.halo.size() - p.h0;
						plan.halo.push_back(J);
					}
					if (local[J] > 65535) return plan;
					plan.lcol[k] = (uint16_t)local[J];
				}
				else
				{
					if (J - r0 > 65535) return plan;
					plan.lcol[k] = (uint16_t)(J - r0);
				}
			}
			p.h1 = (int)plan.halo.size();
			for (int j = p.h0; j < p.h1; ++j) local[plan.halo[j]] = -1;
			if (res_mixed(form))
			{
				// Chunks over the row warps: the widest first, each to the warp with the least to do.
				const int n = p.c1 - p.c0;
				std::vector<int> order(n), load(kResRowWarps, 0);
				std::vector<std::vector<int>> list(kResRowWarps);
				std::iota(order.begin(), order.end(), 0);
				auto slots = [&](int c) { return off[p.c0 + c + 1] - off[p.c0 + c]; };
				std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return slots(a) > slots(b); });
				for (int c : order)
				{
					const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
					load[w] += slots(c) + 4;
					list[w].push_back(c);
				}
				p.warp0 = (int)plan.chunkWarp.size();
				for (const std::vector<int>& l : list)
				{
					plan.chunkWarp.push_back((int)plan.chunkList.size());
					plan.chunkList.insert(plan.chunkList.end(), l.begin(), l.end());
				}
				plan.chunkWarp.push_back((int)plan.chunkList.size());
			}
			plan.parts.push_back(p);
		}
		plan.segPart.push_back((int)plan.parts.size());
		plan.mailWords += res_mail_words(g);
		if (plan.mailWords > (size_t)1 << 24) return plan;
	}
	if (!res_fits(plan, form, smemBudget)) return plan;
	// Longest first: a long system that starts last would be waited for.
	std::vector<double> length(nseg);
	for (int s = 0; s < nseg; ++s)
		length[s] = cost[s] * (200.0 + (off[cut[s].back()] - off[cut[s][0]]) / (double)width[s]);
	std::vector<int> order(nseg);
	std::iota(order.begin(), order.end(), 0);
	std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return length[a] > length[b]; });
	for (int s : order)
		for (int p = plan.segPart[s]; p < plan.segPart[s + 1]; ++p) plan.tasks.push_back(make_int2(p, 0));
	plan.grid = std::min(ctas, (int)plan.tasks.size());
	plan.ok = true;
	return plan;
}

bool res_fits(const ResPlan& plan, int form, int smemBudget)
{
	for (const ResPart& p : plan.parts)
		if (res_layout(form, p.c1 - p.c0, p.h1 - p.h0).mat > smemBudget) return false;
	return true;
}

size_t res_smem(const ResPlan& plan, int form, const std::vector<int>& off, int smemBudget)
{
	long long most = 0;
	for (const ResPart& p : plan.parts)
	{
		const ResLayout L = res_layout(form, p.c1 - p.c0, p.h1 - p.h0);
		most = std::max(most, L.mat + (long long)(off[p.c1] - off[p.c0]) * L.slotBytes);
	}
	return (size_t)std::min<long long>(most, smemBudget);
}

}  // namespace gbfem
