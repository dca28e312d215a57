// Host check of the resident CG's plans (gbfem_plan.cpp) and of the slot and piece arithmetic the kernel does
// with them (gbfem_res.cu, open_share / open_mixed / product), on random SELL matrices: every chunk in one
// share, local columns naming the right rows, shares within the shared memory, every slot multiplied once
// (mixed: every chunk by one warp), cut chunks made of exactly their pieces, every share drawn once with its
// system's others. Prints
// "plan ok" or the first violation.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "gbfem_plan.h"

using namespace gbfem;

#define CHECK(x)                                                           \
	do                                                                     \
		if (!(x))                                                          \
		{                                                                  \
			std::printf("line %d: %s (trial %d)\n", __LINE__, #x, trial);  \
			return 1;                                                      \
		}                                                                  \
	while (0)

namespace {

std::mt19937 rng(1);
int random_int(int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); }

int check_node_parts(int trial)
{
	const int n = random_int(1, 5000), g = random_int(1, std::min((n + 31) / 32, 150));
	std::vector<double> X(3 * n);
	for (double& v : X) v = trial % 3 == 0 ? random_int(0, 4) : rng() / 1e9;
	std::vector<int> w(n), seen(n, 0);
	for (int& v : w) v = random_int(1, 27);
	const auto parts = res_node_parts(X.data(), w, g);
	CHECK((int)parts.size() == g);
	for (int k = 0; k < g; ++k)
	{
		CHECK(!parts[k].empty());
		CHECK(k + 1 == g || parts[k].size() % 32 == 0);
		for (int i : parts[k]) seen[i]++;
	}
	for (int s : seen) CHECK(s == 1);
	return 0;
}

int check_plan(int trial)
{
	const int ctas = 152, budget = 231424;
	int nseg = trial == 7 ? 300 : (trial % 3 == 0 ? 1 : random_int(1, 4));
	std::vector<int> segChunk{0}, off{0}, rcol;
	for (int s = 0; s < nseg; ++s)
	{
		const int nc = nseg == 300 ? random_int(1, 3) : random_int(1, trial % 5 == 0 ? 600 : 40);
		for (int c = 0; c < nc; ++c) off.push_back(off.back() + random_int(1, trial % 4 == 1 ? 3 : 27));
		segChunk.push_back(segChunk.back() + nc);
	}
	for (int s = 0; s < nseg; ++s)
		for (int c = segChunk[s]; c < segChunk[s + 1]; ++c)
			for (int k = 32 * off[c]; k < 32 * off[c + 1]; ++k)
				rcol.push_back(std::max(32 * segChunk[s], std::min(32 * segChunk[s + 1] - 1, 32 * c + k % 32 + random_int(-200, 200))));
	for (int form = 0; form < kResForms; ++form)
	{
		std::vector<long long> weight(nseg, 0);
		std::vector<int> chunks(nseg);
		for (int s = 0; s < nseg; ++s)
		{
			chunks[s] = segChunk[s + 1] - segChunk[s];
			for (int c = segChunk[s]; c < segChunk[s + 1]; ++c) weight[s] += res_chunk_weight(off[c + 1] - off[c]);
		}
		const std::vector<int> width = res_widths(form, 1.7, weight, chunks, std::vector<double>(nseg, 1.0), ctas, budget);
		std::vector<std::vector<int>> cut(nseg);
		for (int s = 0; s < nseg; ++s)
		{
			cut[s] = res_cut(off, segChunk[s], segChunk[s + 1], width[s]);
			CHECK((int)cut[s].size() == width[s] + 1);
		}
		const ResPlan plan = res_plan(form, cut, off, rcol, std::vector<double>(nseg, 1.0), ctas, budget);
		CHECK(plan.ok);
		int next = 0;
		for (const ResPart& p : plan.parts)
		{
			CHECK(p.c0 == next && p.c1 > p.c0);
			next = p.c1;
			const ResLayout L = res_layout(form, p.c1 - p.c0, p.h1 - p.h0);
			CHECK(L.mat <= budget && L.mat % 128 == 0 && L.loc % 16 == 0 && L.own % 8 == 0 && L.part % 8 == 0);
			for (int k = 32 * off[p.c0]; k < 32 * off[p.c1]; ++k)
			{
				const int lc = plan.lcol[k];
				CHECK(lc < L.nLoc);
				CHECK((lc < L.nOwn ? 32 * p.c0 + lc : plan.halo[p.h0 + lc - L.nOwn]) == rcol[k]);
			}
			// The kernel's split of the share's slots over its warps, with some or all of them kept.
			const long long slots = off[p.c1] - off[p.c0];
			int kept = (int)std::min<long long>(slots, (budget - L.mat) / L.slotBytes);
			if (trial % 2) kept = kept * random_int(0, 99) / 100;
			if (res_mixed(form))
			{
				// Whole chunks a warp; every chunk keeps its leading slots, one after the other.
				std::vector<int> seen(L.nCh, 0);
				for (int w = 0; w < kResRowWarps; ++w)
					for (int j = plan.chunkWarp[p.warp0 + w]; j < plan.chunkWarp[p.warp0 + w + 1]; ++j) seen[plan.chunkList[j]]++;
				for (int s : seen) CHECK(s == 1);
				auto keptAt = [&](int c) { return (int)((long long)(off[p.c0 + c] - off[p.c0]) * kept / slots); };
				for (int c = 0; c < L.nCh; ++c)
				{
					const int n = keptAt(c + 1) - keptAt(c);
					CHECK(n >= 0 && n <= off[p.c0 + c + 1] - off[p.c0 + c]);
				}
				CHECK(keptAt(0) == 0 && keptAt(L.nCh) == kept && L.pieces + 4 * (L.nCh + 1) <= L.halo);
				continue;
			}
			const int nw = (int)std::min<long long>(slots, L.nCh <= 2 ? 7 : (L.nCh <= 4 ? 10 : kResRowWarps));
			auto first = [&](int w) { return w >= nw ? (int)slots : (int)(w * slots / nw); };
			auto keptFirst = [&](int w) { return w >= nw ? kept : w * kept / nw; };
			auto at = [&](int c) { return off[p.c0 + c] - off[p.c0]; };
			std::vector<int> hit(slots, 0), owner(kResPieces, -1), wholeBy(L.nCh, -1), keptHit(kept, 0);
			std::vector<long long> sum(kResPieces, 0), whole(L.nCh, 0);
			for (int w = 0; w < kResRowWarps; ++w)
			{
				int s = first(w);
				const int s1 = first(w + 1), sk = s + std::min(keptFirst(w + 1) - keptFirst(w), s1 - s);
				if (s >= s1) continue;
				int c0 = 0;
				while (c0 + 1 < L.nCh && at(c0 + 1) <= s) ++c0;
				for (int c = c0; s < s1; ++c)
				{
					const int e = std::min(s1, at(c + 1)), s0 = s;
					long long t = 0;
					for (; s < e; ++s)
					{
						hit[s]++;
						t += s + 1;
						if (s >= sk) continue;
						const int k = keptFirst(w) + s - first(w);
						CHECK(k >= 0 && k < kept && !keptHit[k]++);
					}
					if (e - s0 == at(c + 1) - at(c))
					{
						CHECK(wholeBy[c] < 0);
						wholeBy[c] = w;
						whole[c] = t;
						continue;
					}
					const int piece = 2 * w + (c == c0 ? 0 : 1);
					CHECK(owner[piece] < 0);
					owner[piece] = c;
					sum[piece] = t;
				}
			}
			for (int h : hit) CHECK(h == 1);
			for (int c = 0; c < L.nCh; ++c)
			{
				long long want = 0, got = 0;
				for (int s = at(c); s < at(c + 1); ++s) want += s + 1;
				const int w0 = (int)(((long long)(at(c) + 1) * nw - 1) / slots), w1 = (int)(((long long)at(c + 1) * nw - 1) / slots);
				if (w0 == w1)
				{
					CHECK(wholeBy[c] == w0);
					got = whole[c];
				}
				else
				{
					const int f0 = 2 * w0 + (first(w0) < at(c) ? 1 : 0);
					CHECK(owner[f0] == c);
					got = sum[f0];
					for (int w = w0 + 1; w <= w1; ++w)
					{
						CHECK(owner[2 * w] == c);
						got += sum[2 * w];
					}
				}
				CHECK(want == got);
			}
		}
		CHECK(next == segChunk.back());
		size_t mail = 0;
		for (int s = 0; s < nseg; ++s)
		{
			CHECK((size_t)plan.parts[plan.segPart[s]].mail0 == mail);
			mail += res_mail_words(width[s]);
		}
		CHECK(mail == plan.mailWords);
		std::vector<int> drawn(plan.parts.size(), 0);
		for (size_t t = 0; t < plan.tasks.size(); ++t)
		{
			const int q = plan.tasks[t].x;
			drawn[q]++;
			CHECK(plan.parts[q].rank == 0 || plan.tasks[t - 1].x == q - 1);
			CHECK(plan.parts[q].g <= plan.grid);
		}
		for (int d : drawn) CHECK(d == 1);
	}
	return 0;
}

}  // namespace

int main()
{
	for (int trial = 0; trial < 300; ++trial)
		if (check_node_parts(trial)) return 1;
	for (int trial = 0; trial < 60; ++trial)
		if (check_plan(trial)) return 1;
	std::printf("plan ok\n");
	return 0;
}
