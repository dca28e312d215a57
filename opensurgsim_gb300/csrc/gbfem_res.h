// gbfem_res.h -- resident CG: systems whose matrix stays in the SMs' shared memory (declarations).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "gbfem_pcg.h"

namespace gbfem {

constexpr int kResRowWarps = 15;  // warps of a CTA that own rows; one more sums and talks to the other CTAs
constexpr int kResThreads = 32 * (kResRowWarps + 1);
constexpr int kResCluster = 16;    // CTAs of a system that may run as one cluster
constexpr int kResMaxGroup = 160;  // CTAs one system may spread over

// One CTA's share of a system: a contiguous range of SELL-32 chunks, the rows of other CTAs its blocks
// refer to (halo), and the system's mailbox.
struct ResPart
{
	int seg, rank, g;   // system, this share's place among its g shares
	int c0, c1;         // chunks
	int h0, h1;         // entries of ResArgs::halo
	int mail0;          // first mailbox word of the system
	int warp0;          // mixed forms: the share's entries of ResArgs::chunkWarp (a row warp each, and the end)
};

// 16-byte words that carry their own tag: CTAs exchange rows and sums through them with relaxed
// single-copy-atomic 128-bit accesses, so no fence orders an exchange (ResArgs::epoch).
struct alignas(16) ResWord
{
	unsigned a, b, c, tag;
};

struct ResCtl
{
	unsigned epoch;     // tags of this launch start above it
	unsigned maxPhase;  // phases the launch has used so far
	unsigned done;      // CTAs that have finished
	unsigned beat;      // advances while any system iterates
	unsigned ticket;    // next entry of ResArgs::tasks
};

// When a wait has run out: its limit is past on the clock and it has polled kResPolls times (1 ms and more), both since it
// began or since some system of the launch last advanced (ResCtl::beat: a CTA may wait for another that is busy with an
// earlier system). While the GPU runs another program the clock goes on and no CTA of this one does: a wait that
// finds its limit past after such a pause is still polled.
constexpr unsigned kResPolls = 2048;
struct ResPatience
{
	unsigned polls = 0, seen = 0;
	unsigned long long t0 = 0;
	// After a poll: whether to look at the time, after every 128.
	__host__ __device__ bool look() { return (++polls & 127u) == 0; }
	// At time t (ns): whether the wait has run out.
	__host__ __device__ bool over(unsigned long long t, unsigned beat, long long limit)
	{
		if (t0 == 0 || beat != seen)
		{
			t0 = t;
			seen = beat;
			polls = 0;
		}
		return polls >= kResPolls && (long long)(t - t0) > limit;
	}
};

struct ResArgs
{
	const ResPart* parts;
	const int2* tasks;    // {part, right-hand side} in the order CTAs draw them, a system's shares together
	int nTasks;
	const int* off;       // SELL-32 chunk offsets in block columns
	const uint16_t* lcol; // column of a slot as a local row: own rows first, then the halo in list order
	const int* halo;      // row positions
	const int* chunkWarp; // mixed forms: first entry of chunkList of every row warp
	const int* chunkList; // chunks of a share (from its first) by the warp that multiplies them
	const int* perm;      // row position -> node (or scalar row), -1 on padding rows
	const int* segMaxIter;  // per system, or null: maxIter
	int maxIter, smemBudget;
	int cluster;          // whether the launch is one system's CTAs as one cluster
	float nearFraction;   // mixed forms: part of the slots beyond shared memory that L2 is to keep
	double tol, drop;
	long long timeoutNs;
	ResWord* mail;        // mailboxes of all systems; right-hand side c uses mail + c * mailStride
	ResWord* rowWords;    // exchanged rows (res_row_words per row and right-hand side)
	size_t mailStride, rowStride;
	ResCtl* ctl;
	SegCtl* seg;          // results per system and right-hand side (segStride apart)
	int* err;
	int segStride;
	size_t vecStride;     // dofs between right-hand sides in b and x
	const double* b;
	double* x;
	const void* val;      // SELL values (float or double)
	const void* invdiag;  // float or double, dof space
	float2* xhl;          // mixed form: the folded solution as float pairs, row space, 3 per row
	double* r64;          // mixed form: the true residual, row space, 3 per row
	float4* own;           // kResMixedFar: p, then x_delta, of every row
	int nrows;
};

// Kernels. kResMixed: FP32 CG with double-float refreshes (Chronopoulos and Gear's recurrences, the
// one-phase schedule of k_pcg_persistent); kResMixedFar: the same with p and x_delta in global memory, for
// shares whose other vectors fill the shared memory; kResF64: Eigen's FP64 CG on FP64 3x3 blocks; kResF64M: the
// same on FP32 blocks (compliance of the mixed form); kResF64S: the same on a scalar FP64 matrix.
enum ResForm : int
{
	kResMixed = 0,
	kResF64 = 1,
	kResF64M = 2,
	kResF64S = 3,
	kResMixedFar = 4,
	kResForms = 5,
};

// Row words per row: mixed {w, w (other parity), t, l, r64 (2)}; FP64 one per element of z.
constexpr int res_row_words(int form)
{
	return form == kResMixed || form == kResMixedFar ? 6 : (form == kResF64S ? 1 : 3);
}
// Mailbox words of a system spread over g CTAs: two parities, g consumers, g producers, two words.
constexpr size_t res_mail_words(int g) { return (size_t)4 * g * g; }

// Dynamic shared memory of one share, in bytes from its start: the fixed part (lists, local and own
// vectors, the partial sums of chunks that warps cut); the matrix takes what is left.
struct ResLayout
{
	int nOwn, nLoc, nCh;
	int offL, pieces, halo, loc, own, part, mat;  // byte offsets
	int slotBytes;                                // matrix values and local columns of one slot (32 rows)
};
__host__ __device__ inline int res_up(int v, int m) { return (v + m - 1) / m * m; }
// Bytes of a local row's vectors (mixed: u, r, s, w as float4; FP64: p, z), of an own row's (p, x_delta, in
// global memory for kResMixedFar; x, r, d, q) and of a row's partial sum.
__host__ __device__ constexpr bool res_mixed(int form) { return form == kResMixed || form == kResMixedFar; }
__host__ __device__ constexpr int res_loc_bytes(int form) { return res_mixed(form) ? 64 : (form == kResF64S ? 16 : 48); }
__host__ __device__ constexpr int res_own_bytes(int form)
{
	return form == kResMixedFar ? 0 : (form == kResMixed || form == kResF64S ? 32 : 96);
}
__host__ __device__ constexpr int res_part_bytes(int form) { return res_mixed(form) ? 0 : (form == kResF64S ? 8 : 24); }
constexpr int kResPieces = 2 * kResRowWarps;  // a warp cuts at most its first and its last chunk
__host__ __device__ inline ResLayout res_layout(int form, int nCh, int nHalo)
{
	ResLayout L;
	L.nCh = nCh;
	L.nOwn = 32 * nCh;
	L.nLoc = L.nOwn + nHalo;
	L.offL = 0;
	L.pieces = 4 * (nCh + 1);
	L.halo = res_up(L.pieces + 4 * (nCh + 1), 16);
	L.loc = L.halo + res_up(4 * nHalo, 16);
	L.own = L.loc + res_loc_bytes(form) * L.nLoc;
	L.part = L.own + res_own_bytes(form) * L.nOwn;
	L.mat = res_up(L.part + kResPieces * 32 * res_part_bytes(form), 128);
	const int blk = form == kResF64S ? 1 : 9, mb = (res_mixed(form) || form == kResF64M) ? 4 : 8;
	L.slotBytes = 32 * blk * mb + 64;
	return L;
}

cudaError_t res_set_max_dynamic_smem(int form, int bytes);
// Whether `ctas` CTAs with this much dynamic shared memory can run as one cluster.
bool res_cluster_fits(int form, int ctas, size_t smem);
cudaError_t res_launch(int form, int grid, size_t smem, const ResArgs& a, cudaStream_t s);

}  // namespace gbfem
