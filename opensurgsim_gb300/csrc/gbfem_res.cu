// gbfem_res.cu -- resident CG: one cooperative launch solves systems whose matrix stays in shared memory.
//
// The launch-per-iteration CG and the persistent CG of gbfem_pcg.cu read the matrix from L2 or HBM in
// every iteration and end every phase at a grid-wide barrier, so a system that does not fill the chip
// spends its time on dependent loads and barriers (1,331 nodes: 46 us an iteration in FP64, 14.5 us a
// phase in the mixed form). Here a system is cut into shares of whole 32-row chunks, spatially compact,
// one CTA of 512 threads per share and SM; a CTA keeps its share of the matrix and its local vectors in
// shared memory for the whole solve (34 MB over the chip), and the CTAs of a system exchange only halo
// rows and dot products.
//
// Exchanges use 16-byte words that carry a tag (the phase): a word is written and read by one relaxed
// 128-bit access, single-copy atomic, so a reader that sees the tag has the data and no fence is needed
// (an all-gather of sums among 16 CTAs: 0.9 us, against 2.2-2.5 us with release/acquire flags and
// 3.4 us for the grid). Every CTA of a system sums the same partials in the same order and takes
// the same decisions; results do not depend on timing. A buffer written in phase k is written again in
// phase k + 2, after its writer has every CTA's sums of phase k + 1, which each CTA sends after it
// has used the words of phase k. Waits end after a time limit (ResArgs::timeoutNs): the launch
// then reports an error and returns.
//
// Systems of a batch are independent: each is solved by its own group of CTAs (as many as its matrix
// needs), groups side by side and, when they outnumber the SMs, one after the other.
//
// Solve times, before (gbfem_pcg.cu's, of one launch an iteration or persistent) and here: FP64 80 nodes 2.9
// and 0.34 ms, 1,331 nodes 3.3 and 0.49, 29,184 nodes 4.1 and 1.18, 24 meshes 10.4 and 3.0; mixed 1,331
// nodes 1.40 and 0.23, 18,081 nodes 1.93 and 0.38, 270,641 nodes (410 iterations) 18.3 and 12.5, 64 meshes 15.7
// and 5.0; 12 compliance columns of 1,331 nodes 47 and 0.94; a caller's matrix of 17,280 rows 2.98 and 0.46.
// What bounds them: the waits of an iteration (a sum over CTAs takes 0.5 us in a cluster, 1.2 to 1.8 us through L2;
// FP64 has two an iteration of 4.5 to 15 us, mixed one of 2.7 to 4.5), the FP64 rate (64 cycles an instruction
// of a warp) in FP64 products and sums, and the L2 and HBM reads of what does not fit in shared memory in large
// systems.

#include <cfloat>
#include <cstdint>
#include <type_traits>

#include "gbfem_res.h"

namespace gbfem {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// ---- tagged words ---------------------------------------------------------------------------------------
__device__ __forceinline__ void st_word(ResWord* p, unsigned a, unsigned b, unsigned c, unsigned tag)
{
	const unsigned long long lo = ((unsigned long long)b << 32) | a, hi = ((unsigned long long)tag << 32) | c;
	asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" : : "l"(p),
				 "l"(lo), "l"(hi)
				 : "memory");
}

__device__ __forceinline__ ResWord ld_word(const ResWord* p)
{
	unsigned long long lo, hi;
	asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
				 : "=l"(lo), "=l"(hi)
				 : "l"(p)
				 : "memory");
	ResWord w;
	w.a = (unsigned)lo;
	w.b = (unsigned)(lo >> 32);
	w.c = (unsigned)hi;
	w.tag = (unsigned)(hi >> 32);
	return w;
}

__device__ __forceinline__ unsigned long long global_ns()
{
	unsigned long long t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}

// Bound on one wait: after every 128 polls, whether another wait has given up or this one's time has run out (then the
// launch's error flag is set).
struct Patience
{
	ResPatience time;
	__device__ __forceinline__ bool lost(const ResArgs& a)
	{
		if (!time.look()) return false;
		const unsigned long long t = global_ns();
		if (*(volatile int*)a.err) return true;
		if (!time.over(t, *(volatile unsigned*)&a.ctl->beat, a.timeoutNs)) return false;
		atomicExch(a.err, 1);
		return true;
	}
};

// ---- double-float scalars ---------------------------------------------------------------------------------
// a + b = s + e exactly (Knuth); the _rn intrinsics keep the compiler from contracting it.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
	s = __fadd_rn(a, b);
	const float bb = __fsub_rn(s, a);
	e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
// Unevaluated pair h + l (~2^-46 relative). Sums and the CG scalars of the mixed form are held so: an
// FP64 instruction takes 64 cycles of a scheduler here and an FP64 division 565 cycles.
// The exponents are FP32's: talk_mixed scales what the matrix's units could put near its ends.
struct Pair
{
	float h, l;
};
__device__ __forceinline__ Pair pair(float h, float l)
{
	const float s = __fadd_rn(h, l);
	return {s, __fadd_rn(__fsub_rn(h, s), l)};
}
__device__ __forceinline__ Pair operator+(Pair a, Pair b)
{
	float s, e;
	two_sum(a.h, b.h, s, e);
	return {s, __fadd_rn(e, __fadd_rn(a.l, b.l))};  // l stays far below h: renormalised where it matters
}
__device__ __forceinline__ Pair operator-(Pair a, Pair b)
{
	const Pair d = a + Pair{-b.h, -b.l};
	return pair(d.h, d.l);
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b)
{
	const float p = __fmul_rn(a.h, b.h);
	return pair(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p))));
}
__device__ __forceinline__ Pair operator/(Pair a, Pair b)
{
	const float q = __fdiv_rn(a.h, b.h);
	const float p = __fmul_rn(q, b.h);
	const float r = __fadd_rn(__fsub_rn(__fsub_rn(a.h, p), __fmaf_rn(q, b.h, -p)), __fmaf_rn(-q, b.l, a.l));
	return pair(q, __fdiv_rn(r, b.h));
}
__device__ __forceinline__ Pair to_pair(double v)
{
	const float h = __double2float_rn(v);
	return {h, __double2float_rn(v - double(h))};
}
__device__ __forceinline__ Pair shfl_xor(Pair v, int o)
{
	return {__shfl_xor_sync(kFull, v.h, o), __shfl_xor_sync(kFull, v.l, o)};
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
	return v;
}

// ---- one share --------------------------------------------------------------------------------------------
// The row warps own the rows and the matrix; one more warp sums, talks to the other CTAs and takes the CG
// decisions, so the scalars' registers and latencies stay out of the row code. Barriers: 1 (sums ready:
// the row warps arrive, the talking warp waits), 2 (scalars ready: the other way), 3 (row warps), 4 (next
// share). A wait that gives up sets `bad`; the talking warp alone turns that into mode 3, which every row
// warp reads after barrier 2, so all of them leave a share at the same place.

struct Shared
{
	int bad;    // a wait gave up
	unsigned phases;
	int task;
	int mode;   // next phase: 0 CG step, 1 true residual, 2 rescale, 3 finished
	int tiny;   // FP64: whether the solve runs on kUp times the right-hand side
	float al, be, as, ratio;
	double inv;   // 1 / s
	double alpha, beta;
	float2 red[3][16];
	double dsum[2][16];
};
__shared__ Shared sh;
extern __shared__ __align__(128) unsigned char smem[];
template <typename T>
__device__ __forceinline__ T* shm(int offset)
{
	return reinterpret_cast<T*>(smem + offset);
}

constexpr int kRowThreads = 32 * kResRowWarps;

__device__ __forceinline__ void rows_sync() { asm volatile("bar.sync 3, %0;" : : "n"(kRowThreads) : "memory"); }
__device__ __forceinline__ void sums_ready() { asm volatile("bar.arrive 1, %0;" : : "n"(kResThreads) : "memory"); }
__device__ __forceinline__ void sums_wait() { asm volatile("bar.sync 1, %0;" : : "n"(kResThreads) : "memory"); }
__device__ __forceinline__ void scalars_ready() { asm volatile("bar.arrive 2, %0;" : : "n"(kResThreads) : "memory"); }
__device__ __forceinline__ void share_draw() { asm volatile("bar.sync 4, %0;" : : "n"(kResThreads) : "memory"); }
__device__ __forceinline__ void scalars_wait() { asm volatile("bar.sync 2, %0;" : : "n"(kResThreads) : "memory"); }

template <int kForm>
struct Types
{
	using M = double;   // matrix values
	using V = double;   // vectors
	using D = double;   // Jacobi inverse as given
	static constexpr int bs = 3;
};
template <>
struct Types<kResMixed>
{
	using M = float;
	using V = float;
	using D = float;
};
template <>
struct Types<kResMixedFar> : Types<kResMixed>
{
};
template <>
struct Types<kResF64M>
{
	using M = float;
	using V = double;
	using D = float;
	static constexpr int bs = 3;
};
template <>
struct Types<kResF64S>
{
	using M = double;
	using V = double;
	using D = double;
	static constexpr int bs = 1;
};

// What a row warp knows of its share. FP64 forms: row warp w multiplies the slots [first(w), first(w + 1)) of
// the share's slots in chunk order; the leading ones of each warp's range are in shared memory (all of them
// when the share fits), the others are read from global memory in every product. A chunk that several warps
// cut gets one partial sum per warp; a chunk of one warp's goes straight to its rows.
struct Share
{
	ResLayout L;
	int c0, nHalo;
	int s, sk, s1, c;      // this warp's slots [s, s1), of which [s, sk) are kept; the chunk of s
	int valKept, colKept;  // shared offsets such that slot k is at offset + k * (its size)
	const unsigned char *val, *col;  // the same in global memory
};

// Warps that share the product: an FP64 instruction takes 64 cycles of a scheduler and 19 of the SM, so few warps
// saturate it, and every piece more a chunk is cut into costs its rows an FP64 add (solves of 1,331 nodes, one chunk a
// share: 0.508 ms with 4 warps, 0.485 with 7, 0.494 with 10; of 4,913, two to four chunks: 0.667 with 4 and 8, 0.623
// with 7 and 10).
__device__ __forceinline__ int product_warps(int nCh)
{
	return nCh <= 2 ? 7 : (nCh <= 4 ? 10 : kResRowWarps);
}
__device__ __forceinline__ int part_first(int w, int n, int nw) { return w >= nw ? n : w * n / nw; }

template <int kForm>
__device__ __forceinline__ Share open_share(const ResArgs& a, const ResPart& p)
{
	using M = typename Types<kForm>::M;
	constexpr int bs = Types<kForm>::bs;
	constexpr int kVal = bs * bs * 32 * (int)sizeof(M);  // bytes of a slot's values
	const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
	Share S;
	S.L = res_layout(kForm, p.c1 - p.c0, p.h1 - p.h0);
	S.c0 = p.c0;
	S.nHalo = p.h1 - p.h0;
	const int k0 = a.off[p.c0];
	const int slots = a.off[p.c1] - k0;
	const int mat = S.L.mat;
	const int kept = max(0, min(slots, (a.smemBudget - mat) / S.L.slotBytes));
	const int nw = min(slots, product_warps(S.L.nCh));
	int* offL = shm<int>(S.L.offL);
	int* pieces = shm<int>(S.L.pieces);
	int* halo = shm<int>(S.L.halo);
	for (int i = threadIdx.x; i <= S.L.nCh; i += kRowThreads) offL[i] = a.off[p.c0 + i] - k0;
	// The warp holding slot s is the largest w with first(w) <= s: a chunk's first and last warp. A chunk cut
	// by warps has a piece in each, piece 2w of warp w when the chunk is its first, else 2w + 1.
	for (int i = threadIdx.x; i < S.L.nCh; i += kRowThreads)
	{
		const int s = a.off[p.c0 + i] - k0, e = a.off[p.c0 + i + 1] - k0;
		const int w0 = ((s + 1) * nw - 1) / slots, w1 = (e * nw - 1) / slots;
		pieces[i] = (2 * w0 + (part_first(w0, slots, nw) < s ? 1 : 0)) + 256 * w1 + (w0 == w1 ? 65536 : 0);
	}
	for (int i = threadIdx.x; i < S.nHalo; i += kRowThreads) halo[i] = a.halo[p.h0 + i];
	S.s = part_first(w, slots, nw);
	S.s1 = part_first(w + 1, slots, nw);
	const int d0 = part_first(w, kept, nw), n = min(part_first(w + 1, kept, nw) - d0, S.s1 - S.s);
	S.sk = S.s + n;
	S.val = static_cast<const unsigned char*>(a.val) + (size_t)k0 * kVal;
	S.col = reinterpret_cast<const unsigned char*>(a.lcol) + (size_t)k0 * 64;
	S.valKept = mat + (d0 - S.s) * kVal;
	S.colKept = mat + kept * kVal + (d0 - S.s) * 64;
	int lo = p.c0, hi = p.c1 - 1;  // chunk of slot s: the last with offset <= s (chunks are not empty)
	while (lo < hi)
	{
		const int mid = (lo + hi + 1) >> 1;
		if (a.off[mid] - k0 <= S.s)
			lo = mid;
		else
			hi = mid - 1;
	}
	S.c = lo - p.c0;
	// The kept part of this warp's slots: contiguous in global memory, 16 bytes a load.
	const uint4* src = reinterpret_cast<const uint4*>(S.val + (size_t)S.s * kVal);
	uint4* dst = shm<uint4>(mat + d0 * kVal);
#pragma unroll 4
	for (int i = lane; i < n * (kVal / 16); i += 32) dst[i] = __ldg(&src[i]);
	const uint4* csrc = reinterpret_cast<const uint4*>(S.col + (size_t)S.s * 64);
	uint4* cdst = shm<uint4>(mat + kept * kVal + d0 * 64);
	for (int i = lane; i < n * 4; i += 32) cdst[i] = __ldg(&csrc[i]);
	return S;
}

// Global row position of local row i.
__device__ __forceinline__ int row_of(const Share& S, int i)
{
	return i < S.L.nOwn ? 32 * S.c0 + i : shm<int>(S.L.halo)[i - S.L.nOwn];
}

// Every chunk piece of this warp's slots: acc.begin(), acc.run(values, columns, slots) over the kept and
// the global ones, then acc.whole(chunk) or acc.cut(piece).
template <int kForm, typename Acc>
__device__ __forceinline__ void product(const Share& S, Acc& acc)
{
	using M = typename Types<kForm>::M;
	const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int* offL = shm<int>(S.L.offL);
	int s = S.s;
	for (int c = S.c; s < S.s1; ++c)
	{
		const int e = min(S.s1, offL[c + 1]), s0 = s;
		acc.begin();
		const int ek = min(e, S.sk);
		if (s < ek)
		{
			acc.template run<false>(shm<M>(S.valKept) + lane, shm<uint16_t>(S.colKept) + lane, s, ek);
			s = ek;
		}
		if (s < e)
		{
			acc.template run<true>(reinterpret_cast<const M*>(S.val) + lane, reinterpret_cast<const uint16_t*>(S.col) + lane,
								   s, e);
			s = e;
		}
		if (e - s0 == offL[c + 1] - offL[c])
			acc.whole(c);
		else
			acc.cut(2 * w + (c == S.c ? 0 : 1));
	}
}

// y = A u on the local rows' u (bs doubles a row: a stride of 24 bytes has no bank conflicts).
template <int kForm>
struct AccMul
{
	using M = typename Types<kForm>::M;
	using V = typename Types<kForm>::V;
	static constexpr int bs = Types<kForm>::bs;
	static constexpr int kVal = bs * bs * 32;
	int u, out, part;  // shared offsets of u, of the own rows' y and of the cut chunks' partials
	V y[bs];
	__device__ __forceinline__ void begin()
	{
#pragma unroll
		for (int i = 0; i < bs; ++i) y[i] = V(0);
	}
	template <bool kGlobal>
	__device__ __forceinline__ void run(const M* v, const uint16_t* col, int s, int e)
	{
#pragma unroll 2
		for (; s < e; ++s)
		{
			const int J = kGlobal ? (int)__ldg(&col[(size_t)s * 32]) : (int)col[s * 32];
			M m[bs * bs];
#pragma unroll
			for (int j = 0; j < bs * bs; ++j) m[j] = kGlobal ? __ldg(&v[(size_t)s * kVal + 32 * j]) : v[s * kVal + 32 * j];
			V x[bs];
#pragma unroll
			for (int j = 0; j < bs; ++j) x[j] = shm<V>(u)[bs * J + j];
#pragma unroll
			for (int i = 0; i < bs; ++i)
#pragma unroll
				for (int j = 0; j < bs; ++j) y[i] = fma(V(m[i * bs + j]), x[j], y[i]);
		}
	}
	__device__ __forceinline__ void put(int base, int at)
	{
#pragma unroll
		for (int i = 0; i < bs; ++i) shm<V>(base)[bs * at + i] = y[i];
	}
	__device__ __forceinline__ void whole(int chunk) { put(out, chunk * 32 + (threadIdx.x & 31)); }
	__device__ __forceinline__ void cut(int piece) { put(part, piece * 32 + (threadIdx.x & 31)); }
};

// Waits for N words with this tag, given by their addresses.
template <int N>
__device__ __forceinline__ void wait_words(const ResArgs& a, const ResWord* const (&p)[N], unsigned tag, ResWord (&w)[N])
{
	Patience wait;
	for (;;)
	{
		bool all = true;
#pragma unroll
		for (int k = 0; k < N; ++k) w[k] = ld_word(p[k]);
#pragma unroll
		for (int k = 0; k < N; ++k) all = all && w[k].tag == tag;
		if (all) break;
		if (wait.lost(a))
		{
			sh.bad = 1;
			break;
		}
	}
}

// Row warps: waits for `words` of every halo element (n of them, word e at words[at(e)]) and stores them by
// put(e, word); two elements a thread are in flight while there are two.
template <int NW, typename A, typename F>
__device__ __forceinline__ void fetch(const ResArgs& a, int n, const ResWord* words, unsigned tag, A at, F put)
{
	int j = threadIdx.x;
#pragma unroll 1
	for (; j + kRowThreads < n; j += 2 * kRowThreads)
	{
		const ResWord *q = words + at(j), *q2 = words + at(j + kRowThreads), *p[2 * NW];
		ResWord w[2 * NW], u[NW];
#pragma unroll
		for (int k = 0; k < NW; ++k) p[k] = q + (size_t)k * a.nrows, p[NW + k] = q2 + (size_t)k * a.nrows;
		wait_words(a, p, tag, w);
#pragma unroll
		for (int k = 0; k < NW; ++k) u[k] = w[k];
		put(j, u);
#pragma unroll
		for (int k = 0; k < NW; ++k) u[k] = w[NW + k];
		put(j + kRowThreads, u);
	}
	if (j < n)
	{
		const ResWord *q = words + at(j), *p[NW];
		ResWord u[NW];
#pragma unroll
		for (int k = 0; k < NW; ++k) p[k] = q + (size_t)k * a.nrows;
		wait_words(a, p, tag, u);
		put(j, u);
	}
}

// The halo rows of a share, NW words a row (word k of row rs at rows[k * nrows + rs]): put(local row, words).
template <int NW, typename S_, typename F>
__device__ __forceinline__ void fetch_halo(const ResArgs& a, const S_& S, const ResWord* rows, unsigned tag, F put)
{
	const int* halo = shm<int>(S.L.halo);
	fetch<NW>(a, S.nHalo, rows, tag, [&](int j) { return halo[j]; },
			  [&](int j, const ResWord(&w)[NW]) { put(S.L.nOwn + j, w); });
}

// The halo rows of a share element by element, bs words a row: put(local element, word).
template <int bs, typename F>
__device__ __forceinline__ void fetch_words(const ResArgs& a, const Share& S, const ResWord* words, unsigned tag, F put)
{
	const int* halo = shm<int>(S.L.halo);
	fetch<1>(a, bs * S.nHalo, words, tag, [&](int j) { return bs * halo[j / bs] + j % bs; },
			 [&](int j, const ResWord(&w)[1]) { put(bs * S.L.nOwn + j, w[0]); });
}

// Row warps, the first `warps` of which have rows: leaves the warp's FP64 sums of NV (1 or 2) values a thread
// for the talking warp. An FP64 add takes 64 cycles whatever its lanes do, so two values are summed in the two
// halves of a warp.
template <int NV>
__device__ __forceinline__ void leave_f64(int warps, const double (&v)[NV])
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	if (warp >= warps) return;  // no rows
	const bool upper = lane >= 16;
	double t = v[0];
	if (NV == 2)
	{
		t = upper ? v[NV - 1] : v[0];
		t += __shfl_xor_sync(kFull, upper ? v[0] : v[NV - 1], 16);
	}
#pragma unroll
	for (int o = NV == 2 ? 8 : 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
	if ((lane & 15) == 0 && (NV == 2 || !upper)) sh.dsum[lane >> 4][warp] = t;
}

// ---- the talking warp ------------------------------------------------------------------------------------------------
template <bool kCluster>  // whether the system is one cluster (send, receive)
struct Talk
{
	int g, nSums;       // CTAs of the system; row warps with rows
	int rank;           // this CTA's place
	ResWord* in;        // this CTA's mailbox (parity 0)
	ResWord* out;       // this CTA's words in CTA 0's mailbox
	int inStep, parity; // words from one consumer's mailbox to the next; from parity 0 to parity 1
};
template <bool kCluster>
__device__ __forceinline__ Talk<kCluster> open_talk(const ResArgs& a, const ResPart& p, int rhs, int warpsPerChunk)
{
	Talk<kCluster> T;
	T.g = p.g;
	T.rank = p.rank;
	T.nSums = min(kResRowWarps, warpsPerChunk * (p.c1 - p.c0));
	ResWord* mail = a.mail + p.mail0 + (size_t)rhs * a.mailStride;
	T.inStep = 2 * p.g;
	T.parity = 2 * p.g * p.g;
	T.in = mail + p.rank * T.inStep;
	T.out = mail + 2 * p.rank;
	return T;
}

// ---- a system in one cluster ------------------------------------------------------------------------------
// Systems of up to kResCluster CTAs run as one thread-block cluster and leave their sums in one another's shared
// memory: two words from every CTA, whose arrival an mbarrier counts, instead of words that travel through L2 and
// are polled for (solves of 80 nodes in FP64: 0.353 ms, through L2 0.380; 392 nodes 0.396 and 0.470; mixed 1,331
// nodes 0.231 and 0.265).
__shared__ ResWord clusterMail[2][kResCluster][2];  // by phase parity, CTA, word
__shared__ __align__(8) unsigned long long clusterBar[2];
__device__ __forceinline__ unsigned shared_address(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned remote_address(unsigned own, int cta)
{
	unsigned a;
	asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(own), "r"(cta));
	return a;
}
__device__ __forceinline__ void cluster_sync()
{
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" : : : "memory");
}

// Sends word {a, b, c} of the lanes 0-15 (0) and 16-31 (1; the same in every lane of a half) to every CTA of the system.
template <bool kCluster>
__device__ __forceinline__ void send(const Talk<kCluster>& T, unsigned ph, unsigned tag, unsigned a, unsigned b, unsigned c)
{
	const int lane = threadIdx.x & 31;
	if constexpr (kCluster)
	{
		const unsigned bar = shared_address(&clusterBar[ph & 1]);
		if (lane == 0)
			asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" : : "r"(bar), "r"(32 * T.g) : "memory");
		if ((lane & 15) < T.g)
			asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" : :
						 "r"(remote_address(shared_address(&clusterMail[ph & 1][T.rank][lane >> 4]), lane & 15)), "r"(a), "r"(b),
						 "r"(c), "r"(tag), "r"(remote_address(bar, lane & 15))
						 : "memory");
		return;
	}
	ResWord* box = T.out + ((ph & 1) ? T.parity : 0) + (lane & 15) * T.inStep + (lane >> 4);
#pragma unroll 1
	for (int j = lane & 15; j < T.g; j += 16, box += 16 * T.inStep) st_word(box, a, b, c, tag);
}

// Waits for every CTA's words of this phase, word 0 in lanes 0-15 and word 1 in lanes 16-31; use(word) is
// called for the CTAs lane % 16, lane % 16 + 16, ... in order. A poll loads the R words a lane needs of up to
// 16 R CTAs and no more: with eight for every system a solve of 80 nodes took 0.469 ms, with four 0.415.
template <int R, typename F>
__device__ __forceinline__ bool receive_words(const ResArgs& a, const ResWord* box, int n, unsigned tag, F use)
{
	ResWord w[R];
	Patience wait;
	for (;;)
	{
#pragma unroll
		for (int r = 0; r < R; ++r) w[r] = ld_word(box + (r < R - 1 || 16 * r < n ? 32 * r : 0));
		bool all = true;
#pragma unroll
		for (int r = 0; r < R; ++r) all = all && w[r].tag == tag;
		if (__all_sync(kFull, all || n <= 0)) break;
		if (__any_sync(kFull, wait.lost(a)))
		{
			sh.bad = 1;
			return false;
		}
	}
#pragma unroll
	for (int r = 0; r < R; ++r)
		if (16 * r < n) use(w[r]);
	return true;
}
// Whether every CTA's 32 bytes of phase ph, the (ph - 1) / 2-th of its parity's barrier, are here.
__device__ __forceinline__ bool arrived(unsigned ph)
{
	const unsigned bar = shared_address(&clusterBar[ph & 1]), parity = ((ph - 1) >> 1) & 1u;
	unsigned done;
	asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
				 : "=r"(done)
				 : "r"(bar), "r"(parity)
				 : "memory");
	return done != 0u;
}
template <bool kCluster, typename F>
__device__ __forceinline__ void receive(const ResArgs& a, const Talk<kCluster>& T, unsigned ph, unsigned tag, F use)
{
	const int lane = threadIdx.x & 31, j = lane & 15;
	if constexpr (kCluster)
	{
		Patience wait;
		for (;;)
		{
			if (__all_sync(kFull, arrived(ph))) break;
			if (__any_sync(kFull, wait.lost(a)))
			{
				sh.bad = 1;
				return;
			}
		}
		if (j < T.g) use(clusterMail[ph & 1][j][lane >> 4]);
		return;
	}
	const ResWord* box = T.in + ((ph & 1) ? T.parity : 0) + (lane >> 4);
#pragma unroll 1
	for (int first = 0; first < T.g; first += 64)
	{
		// Lanes past the last CTA read CTA 0's word (first, in a later batch) and leave it out.
		const int n = T.g - first - j;
		const ResWord* from = box + 2 * (n > 0 ? first + j : 0);
		const int rounds = min(4, (T.g - first + 15) / 16);
		bool ok;
		if (rounds == 1)
			ok = receive_words<1>(a, from, n, tag, use);
		else if (rounds == 2)
			ok = receive_words<2>(a, from, n, tag, use);
		else if (rounds == 3)
			ok = receive_words<3>(a, from, n, tag, use);
		else
			ok = receive_words<4>(a, from, n, tag, use);
		if (!ok) return;
	}
}

// After a solve whose waits gave up, the cluster's CTAs stand at different phases, at most one apart from the last that
// all of them sent: words may still be on their way to a CTA that is done. The talking warp sends what its CTA has
// not sent up to the last phase of any and waits until every word of the last phases has arrived. (A CTA sends in a
// phase only when it has left the one before the last, so a barrier's phase is complete before its next arrival.)
__device__ __noinline__ void settle_cluster()
{
	unsigned rank, g;
	asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
	asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(g));
	const unsigned sent = sh.phases;
	unsigned most = 0;
	for (unsigned j = 0; j < g; ++j)
	{
		unsigned theirs;
		asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(theirs) : "r"(remote_address(shared_address(&sh.phases), (int)j)) : "memory");
		most = max(most, theirs);
	}
	Talk<true> T{};
	T.g = (int)g;
	T.rank = (int)rank;
	const unsigned long long t0 = global_ns();
	for (unsigned ph = sent > 1u ? sent - 1u : 1u; ph <= most; ++ph)
	{
		if (ph > sent) send(T, ph, 0u, 0u, 0u, 0u);
		while (!__all_sync(kFull, arrived(ph)))
			if (__any_sync(kFull, global_ns() - t0 > 1000000000ull)) return;
	}
}

// FP64 sums over the system of the values left by the row warps: the total of value k in v[k] of every
// lane. during() runs while the words travel.
template <int NV, bool kCluster, typename F>
__device__ __forceinline__ void total_f64(const ResArgs& a, const Talk<kCluster>& T, unsigned ph, unsigned tag, double (&v)[NV], F during)
{
	const int lane = threadIdx.x & 31;
	double t = 0.0;
	if ((NV == 2 || lane < 16) && (lane & 15) < T.nSums) t = sh.dsum[lane >> 4][lane & 15];
#pragma unroll
	for (int o = 8; o > 0; o >>= 1)
		if (o < T.nSums) t += __shfl_xor_sync(kFull, t, o);
	if (T.g > 1)
	{
		const unsigned long long u = (unsigned long long)__double_as_longlong(__shfl_sync(kFull, t, lane & 16));
		send(T, ph, tag, (unsigned)u, (unsigned)(u >> 32), 0u);
		during();
		t = 0.0;
		receive(a, T, ph, tag, [&](const ResWord& w) {
			t += __longlong_as_double((long long)(((unsigned long long)w.b << 32) | w.a));
		});
#pragma unroll
		for (int o = 8; o > 0; o >>= 1)
			if (o < T.g) t += __shfl_xor_sync(kFull, t, o);
	}
	else
		during();
#pragma unroll
	for (int k = 0; k < NV; ++k) v[k] = __shfl_sync(kFull, t, 16 * k);
}

// The same for the three sums of an FP32 phase, held as pairs (sh.red).
template <bool kCluster, typename F>
__device__ __forceinline__ void total_pairs(const ResArgs& a, const Talk<kCluster>& T, unsigned ph, unsigned tag, Pair (&v)[3], F during)
{
	const int lane = threadIdx.x & 31, half = lane >> 4, j = lane & 15;
	Pair t{0.f, 0.f}, t2{0.f, 0.f};
	if (j < T.nSums)
	{
		const float2 x = sh.red[half][j], y = sh.red[2][j];
		t = {x.x, x.y};
		t2 = {y.x, y.y};
	}
#pragma unroll
	for (int o = 8; o > 0; o >>= 1)
		if (o < T.nSums)
		{
			t = t + shfl_xor(t, o);
			t2 = t2 + shfl_xor(t2, o);
		}
	if (T.g > 1)
	{
		// Words {r.u, |r|^2 high}, {w.u, |r|^2 low}.
		const int from = lane & 16;  // the lanes that hold the sums whatever the number of warps
		send(T, ph, tag, __float_as_uint(__shfl_sync(kFull, t.h, from)), __float_as_uint(__shfl_sync(kFull, t.l, from)),
			 __float_as_uint(__shfl_sync(kFull, half ? t2.l : t2.h, from)));
		during();
		t = t2 = {0.f, 0.f};
		receive(a, T, ph, tag, [&](const ResWord& w) {
			t = t + Pair{__uint_as_float(w.a), __uint_as_float(w.b)};
			t2 = t2 + Pair{__uint_as_float(w.c), 0.f};
		});
#pragma unroll
		for (int o = 8; o > 0; o >>= 1)
			if (o < T.g)
			{
				t = t + shfl_xor(t, o);
				t2 = t2 + shfl_xor(t2, o);
			}
		t2 = t2 + shfl_xor(t2, 16);
	}
	else
		during();
#pragma unroll
	for (int k = 0; k < 2; ++k) v[k] = {__shfl_sync(kFull, t.h, 16 * k), __shfl_sync(kFull, t.l, 16 * k)};
	v[2] = {__shfl_sync(kFull, t2.h, 0), __shfl_sync(kFull, t2.l, 0)};
}

__device__ __forceinline__ void write_result(const ResArgs& a, const ResPart& p, int rhs, double bb, double rrTrue, int iter,
											 int updates, int converged, int nonfinite)
{
	SegCtl& c = a.seg[p.seg + (size_t)rhs * a.segStride];
	c.bb = bb;
	c.rrTrue = rrTrue;
	c.iter = iter;
	c.updates = updates;
	c.converged = converged;
	c.nonfinite = nonfinite;
	c.done = 1;
}

// Whether a wait of this CTA has given up (the same answer in every lane of the talking warp).
__device__ __forceinline__ bool given_up() { return __any_sync(kFull, *(volatile int*)&sh.bad != 0); }

// The talking warp: publishes the next phase's mode to the row warps.
__device__ __forceinline__ void publish(int mode)
{
	sh.mode = mode;
	__syncwarp();
	scalars_ready();
}

// Counts a phase of the system as progress for waits elsewhere (Patience).
__device__ __forceinline__ void beat(const ResArgs& a, const ResPart& p, unsigned ph)
{
	if (p.rank == 0 && (ph & 15u) < 2 && (threadIdx.x & 31) == 0) atomicAdd(&a.ctl->beat, 1u);
}

// ---- mixed form -----------------------------------------------------------------------------------------
// FP32 CG by Chronopoulos and Gear's recurrences with double-float refreshes: the iteration, stopping
// rule and roundings of k_pcg_persistent<kPcgMixed1>. Each CTA holds u, r, s and the Jacobi inverse of its
// own and its halo rows and advances them all by the same operations, so an iteration exchanges only
// w = A u of the halo rows and one all-gather of sums.

// The talking warp: sums, CG scalars and decisions (the same in every CTA of the system). Returns the phases used.
template <bool kCluster>
__device__ __forceinline__ unsigned talk_mixed(const ResArgs& a, const ResPart p, unsigned base)
{
	const Talk<kCluster> T = open_talk<kCluster>(a, p, 0, 1);
	const int cap = a.segMaxIter ? a.segMaxIter[p.seg] : a.maxIter;
	const int maxLoop = 3 * max(a.maxIter, cap) + 8;
	const float drop = float(a.drop);
	unsigned ph = 1;
	double bb[1], sD = 0.0, threshold, rrTrue;
	Pair sP{}, alpha{1.f, 0.f}, rz{1.f, 0.f}, rzPend{}, ratioP{};
	float rrLast = 0.f, thr32 = 0.f;
	float unit = 1.f;  // what r.u and w.u are scaled by: 1 / r.u stays in FP32's range whatever the matrix's units
	int iter = 0, updates = 0, converged = 0, nonfinite = 0, mode;
	auto rescale = [&](double sNew) {  // r_true ~= s * r
		sD = sNew;
		sP = to_pair(sNew);
		thr32 = __double2float_rn(threshold / (sNew * sNew));
		sh.inv = 1.0 / sNew;
		mode = 2;
	};
	sums_wait();
	total_f64<1>(a, T, ph, base + ph, bb, [] {});
	threshold = fmax(a.tol * a.tol * bb[0], DBL_MIN);
	rrTrue = bb[0];
	nonfinite = !isfinite(bb[0]);
	converged = (bb[0] == 0.0 || bb[0] < threshold) ? 1 : 0;
	if (converged || nonfinite || given_up())
		mode = 3;
	else
		rescale(sqrt(bb[0]));
	publish(mode);
#pragma unroll 1
	for (int it = 0; mode != 3; ++it)
	{
		++ph;
		bool lost = false;  // looked up while words travel; a wait that gives up after that ends the next phase
		beat(a, p, ph);
		sums_wait();
		if (mode == 1)
		{
			double rr[1];
			total_f64<1>(a, T, ph, base + ph, rr, [&] { lost = given_up(); });
			rrTrue = rr[0];
			updates += 1;
			if (rrTrue < threshold)
			{
				converged = 1;  // like Eigen, the converging iteration is not counted
				mode = 3;
			}
			else if (!isfinite(rrTrue) || iter + 1 >= cap)
			{
				nonfinite = !isfinite(rrTrue);
				iter += 1;
				mode = 3;
			}
			else
			{
				const double sNew = sqrt(rrTrue);
				ratioP = to_pair(sD / sNew);
				sh.ratio = ratioP.h;
				rescale(sNew);
			}
		}
		else
		{
			// beta = g / rz and alpha = g / (w.u - beta g / alpha): everything that does not need the
			// new sums is formed while they travel. After a refresh rz is the last one before it, rescaled.
			Pair v[3], rzInv{}, back{};
			const bool first = mode == 2 && updates == 0;
			total_pairs(a, T, ph, base + ph, v, [&] {
				lost = given_up();
				rzInv = Pair{1.f, 0.f} / (mode == 2 ? rzPend * ratioP * ratioP : rz);
				back = rzInv / alpha;
			});
			if (first && !(v[0].h > 0x1p-60f && v[0].h < 0x1p60f))
				unit = __int_as_float(min(max(254 - ((__float_as_int(v[0].h) >> 23) & 255), 1), 253) << 23);
			if (unit != 1.f)
#pragma unroll
				for (int k = 0; k < 2; ++k) v[k] = {unit * v[k].h, unit * v[k].l};
			const Pair gN = pair(v[0].h, v[0].l), dN = pair(v[1].h, v[1].l);
			const float rr = v[2].h + v[2].l;
			if (mode == 0 && (rr < thr32 || rr < drop * rrLast || iter + 1 >= cap))
			{
				rzPend = rz;
				mode = isfinite(rr) ? 1 : 3;  // the true residual of x before the next direction
				nonfinite = mode == 3;
			}
			else
			{
				Pair beta{0.f, 0.f};
				if (first)
					alpha = gN / dN;
				else
				{
					beta = gN * rzInv;
					alpha = gN / (dN - gN * (gN * back));
				}
				nonfinite = !isfinite(rr) || !isfinite(alpha.h);
				sh.al = alpha.h;
				sh.be = beta.h;
				sh.as = (alpha * sP).h;
				if (mode == 2) rrLast = rr;
				if (!first && !nonfinite) iter += 1;  // one that cannot be taken is not counted
				rz = gN;
				mode = nonfinite ? 3 : 0;
			}
		}
		if (it + 1 >= maxLoop || lost) mode = 3;
		publish(mode);
	}
	if (p.rank == 0 && (threadIdx.x & 31) == 0) write_result(a, p, 0, bb[0], rrTrue, iter, updates, converged, nonfinite);
	return ph;
}

// A mixed share's matrix. A chunk belongs to one warp (ResArgs::chunkWarp / chunkList, balanced over the warps),
// whose lanes run through their rows' slots in order, as the persistent solve does: the rows' sums round
// alike. The leading slots of every chunk are kept in shared memory, all of them when the share fits;
// the others are read from global memory in every product.
struct MixedShare
{
	ResLayout L;
	int c0, nHalo, first, last;  // this warp's entries of the chunk list,
	int head;                    // the chunk of the first
	int colKept;                 // shared offset of the kept columns
	unsigned long long policy;   // L2 policy of the slots read in every product
	const float* val;            // the share's first slot
	const uint16_t* col;
};

__device__ __forceinline__ int row_of(const MixedShare& S, int i)
{
	return i < S.L.nOwn ? 32 * S.c0 + i : shm<int>(S.L.halo)[i - S.L.nOwn];
}

template <int kForm>
__device__ __forceinline__ MixedShare open_mixed(const ResArgs& a, const ResPart& p)
{
	const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
	MixedShare S;
	S.L = res_layout(kForm, p.c1 - p.c0, p.h1 - p.h0);
	S.c0 = p.c0;
	S.nHalo = p.h1 - p.h0;
	const int k0 = a.off[p.c0];
	const int slots = a.off[p.c1] - k0;
	const int kept = max(0, min(slots, (a.smemBudget - S.L.mat) / S.L.slotBytes));
	S.val = static_cast<const float*>(a.val) + (size_t)k0 * 288;
	S.col = a.lcol + (size_t)k0 * 32;
	S.colKept = S.L.mat + kept * 1152;
	asm("createpolicy.fractional.L2::evict_normal.L2::evict_first.b64 %0, %1;" : "=l"(S.policy) : "f"(a.nearFraction));
	int* offL = shm<int>(S.L.offL);
	int* keptL = shm<int>(S.L.pieces);  // first kept slot of a chunk: an even share of every chunk's slots
	int* halo = shm<int>(S.L.halo);
	for (int i = tid; i <= S.L.nCh; i += kRowThreads)
	{
		const int o = a.off[p.c0 + i] - k0;
		offL[i] = o;
		keptL[i] = (int)((long long)o * kept / slots);
	}
	for (int i = tid; i < S.nHalo; i += kRowThreads) halo[i] = a.halo[p.h0 + i];
	S.first = a.chunkWarp[p.warp0 + w];
	S.last = a.chunkWarp[p.warp0 + w + 1];
	S.head = S.first < S.last ? a.chunkList[S.first] : 0;
	for (int j = S.first; j < S.last; ++j)
	{
		const int c = a.chunkList[j], o = a.off[p.c0 + c] - k0, o1 = a.off[p.c0 + c + 1] - k0;
		const int d0 = (int)((long long)o * kept / slots), n = (int)((long long)o1 * kept / slots) - d0;
		const uint4* src = reinterpret_cast<const uint4*>(S.val + (size_t)o * 288);
		uint4* dst = shm<uint4>(S.L.mat + d0 * 1152);
#pragma unroll 4
		for (int i = lane; i < n * 72; i += 32) dst[i] = __ldg(&src[i]);
		const uint4* csrc = reinterpret_cast<const uint4*>(S.col + (size_t)o * 32);
		uint4* cdst = shm<uint4>(S.colKept + d0 * 64);
		for (int i = lane; i < n * 4; i += 32) cdst[i] = __ldg(&csrc[i]);
	}
	return S;
}

// Loads of matrix words that no one else reads, with the share's L2 policy: where the matrix does not fit in L2, a
// part of its lines stays and the others leave first, so that part is found there in every product (all of them
// in turn would push one another out; ResArgs::nearFraction).
__device__ __forceinline__ float ld_hint(const float* p, unsigned long long policy)
{
	float v;
	asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(policy));
	return v;
}
__device__ __forceinline__ int ld_hint(const uint16_t* p, unsigned long long policy)
{
	unsigned short v;
	asm("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(policy));
	return v;
}

// A chunk's kept slots.
struct KeptSlots
{
	int val, col;  // shared offsets of this lane's values and columns
	__device__ __forceinline__ int column(int k) const { return shm<uint16_t>(col)[32 * k]; }
	__device__ __forceinline__ void values(int k, float (&m)[9]) const
	{
#pragma unroll
		for (int j = 0; j < 9; ++j) m[j] = shm<float>(val)[288 * k + 32 * j];
	}
};
// A chunk's other slots, in global memory.
struct FarSlots
{
	const float* val;
	const uint16_t* col;
	unsigned long long policy;
	__device__ __forceinline__ int column(int k) const { return ld_hint(&col[32 * k], policy); }
	__device__ __forceinline__ void values(int k, float (&m)[9]) const
	{
#pragma unroll
		for (int j = 0; j < 9; ++j) m[j] = ld_hint(&val[288 * k + 32 * j], policy);
	}
};

// Calls f(slots, n) for the kept and then the other slots of chunk c (this lane's row).
template <typename F>
__device__ __forceinline__ void chunk_slots(const MixedShare& S, int c, F f)
{
	const int lane = threadIdx.x & 31;
	const int o = shm<int>(S.L.offL)[c], o1 = shm<int>(S.L.offL)[c + 1];
	const int d = shm<int>(S.L.pieces)[c], n = shm<int>(S.L.pieces)[c + 1] - d;
	f(KeptSlots{S.L.mat + d * 1152 + 4 * lane, S.colKept + d * 64 + 2 * lane}, n);
	if (n < o1 - o)
		f(FarSlots{S.val + (size_t)(o + n) * 288 + lane, S.col + (size_t)(o + n) * 32 + lane, S.policy}, o1 - o - n);
}

// w = A u for the rows of chunk c, slot by slot with the roundings of k_pcg_persistent's products.
__device__ __forceinline__ void multiply(const MixedShare& S, const float4* U, int c, float& a0, float& a1, float& a2)
{
	chunk_slots(S, c, [&](const auto& slots, int n) {
		// A plain loop: rounds of guarded loads took twice as long in shared memory (19 slots: 2,680 cycles of a
		// warp, here 1,410; 15 warps at once are bound by the shared-memory pipe's 14 words a slot).
		constexpr bool kFar = std::is_same<std::decay_t<decltype(slots)>, FarSlots>::value;
		constexpr int kUnroll = kFar ? 3 : 6;  // far slots: 12.9 ms a solve of 270,641 nodes at 2, 12.6 at 3, 13.4 at 4
#pragma unroll kUnroll
		for (int k = 0; k < n; ++k)
		{
			float m[9];
			const int J = slots.column(k);
			slots.values(k, m);
			const float4 u = U[J];
			a0 += m[0] * u.x + m[1] * u.y + m[2] * u.z;
			a1 += m[3] * u.x + m[4] * u.y + m[5] * u.z;
			a2 += m[6] * u.x + m[7] * u.y + m[8] * u.z;
		}
	});
}

// {x, y, z} of a word.
__device__ __forceinline__ void put_xyz(float4& d, const ResWord& w)
{
	d.x = __uint_as_float(w.a);
	d.y = __uint_as_float(w.b);
	d.z = __uint_as_float(w.c);
}
__device__ __forceinline__ void send_xyz(ResWord* p, float x, float y, float z, unsigned tag)
{
	st_word(p, __float_as_uint(x), __float_as_uint(y), __float_as_uint(z), tag);
}

// Row warps. Local rows: U = {u, d0}, R = {r, d1}, S = {s, d2}, W = {w, -} with d the Jacobi inverse; own
// rows: P = the search direction, X = x_delta.
template <int kForm>
__device__ __forceinline__ void rows_mixed(const ResArgs& a, const ResPart p, unsigned base)
{
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const MixedShare S = open_mixed<kForm>(a, p);
	const int nOwn = S.L.nOwn, nLoc = S.L.nLoc;
	float4* const U = shm<float4>(S.L.loc);
	float4* const R = U + nLoc;
	float4* const Sv = R + nLoc;
	float4* const W = Sv + nLoc;
	const int row0 = 32 * S.c0;
	float4* const P = kForm == kResMixedFar ? a.own + row0 : shm<float4>(S.L.own);
	float4* const X = kForm == kResMixedFar ? P + a.nrows : P + nOwn;
	double* const r64 = a.r64 + 3 * (size_t)row0;  // true residual of the own rows
	const bool alone = p.g == 1;
	unsigned ph = 1;

	// |b|^2 and the Jacobi inverse; x = p = s = 0.
	rows_sync();
	double bb[1] = {0.0};
#pragma unroll 1
	for (int i = tid; i < nLoc; i += kRowThreads)
	{
		const int I = a.perm[row_of(S, i)];
		const float* invdiag = static_cast<const float*>(a.invdiag);
		float d[3];
#pragma unroll
		for (int k = 0; k < 3; ++k)
		{
			d[k] = I >= 0 ? __ldg(&invdiag[3 * I + k]) : 0.f;
			const double bi = (I >= 0 && i < nOwn) ? a.b[3 * I + k] : 0.0;
			bb[0] += bi * bi;
		}
		U[i] = make_float4(0.f, 0.f, 0.f, d[0]);
		R[i] = make_float4(0.f, 0.f, 0.f, d[1]);
		Sv[i] = make_float4(0.f, 0.f, 0.f, d[2]);
		W[i] = make_float4(0.f, 0.f, 0.f, 0.f);
		if (i < nOwn)
		{
			P[i] = X[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
			for (int k = 0; k < 3; ++k) a.xhl[3 * (size_t)(row0 + i) + k] = make_float2(0.f, 0.f);
		}
	}
	leave_f64<1>(S.L.nCh, bb);
	sums_ready();
	scalars_wait();
#pragma unroll 1
	for (;;)
	{
		const int mode = sh.mode;
		if (mode == 3) break;
		++ph;
		const unsigned tag = base + ph;
		if (mode == 1)
		{
			// True residual: x of the local rows as t + l (in U, R), b - A x in double-float, |r|^2 in FP64.
			ResWord* words = a.rowWords + 2 * (size_t)a.nrows;
#pragma unroll 1
			for (int i = tid; i < nOwn; i += kRowThreads)
			{
				const float4 xi = X[i];
				const float xd[3] = {xi.x, xi.y, xi.z};
				float t[3], l[3];
#pragma unroll
				for (int k = 0; k < 3; ++k)
				{
					const float2 x = a.xhl[3 * (size_t)(row0 + i) + k];
					float e;
					two_sum(x.x, xd[k], t[k], e);
					l[k] = __fadd_rn(e, x.y);
				}
				U[i].x = t[0], U[i].y = t[1], U[i].z = t[2];
				R[i].x = l[0], R[i].y = l[1], R[i].z = l[2];
				if (!alone)
				{
					send_xyz(&words[row0 + i], t[0], t[1], t[2], tag);
					send_xyz(&words[(size_t)a.nrows + row0 + i], l[0], l[1], l[2], tag);
				}
			}
			fetch_halo<2>(a, S, words, tag, [&](int i, const ResWord(&v)[2]) {
				put_xyz(U[i], v[0]);
				put_xyz(R[i], v[1]);
			});
			rows_sync();
			// Every product is split exactly by FMA and the row's pair renormalised once a block (the arithmetic of
			// gbfem_pcg.cu's residual_row).
			double rr[1] = {0.0};
			words += 2 * (size_t)a.nrows;
#pragma unroll 1
			for (int j = S.first; j < S.last; ++j)
			{
				const int c = a.chunkList[j], i = 32 * c + lane;
				float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
				chunk_slots(S, c, [&](const auto& slots, int n) {
#pragma unroll 2
					for (int k = 0; k < n; ++k)
					{
						const int J = slots.column(k);
						float v[9];
						slots.values(k, v);
						const float4 tv = U[J], lv = R[J];
						const float x[3] = {tv.x, tv.y, tv.z}, y[3] = {lv.x, lv.y, lv.z};
#pragma unroll
						for (int m = 0; m < 9; ++m)
						{
							const float q = __fmul_rn(v[m], x[m % 3]);
							const float qe = __fmaf_rn(v[m], x[m % 3], -q);
							float hs, he;
							two_sum(hi[m / 3], q, hs, he);
							hi[m / 3] = hs;
							lo[m / 3] = __fadd_rn(lo[m / 3], __fadd_rn(he, __fmaf_rn(v[m], y[m % 3], qe)));
						}
#pragma unroll
						for (int m = 0; m < 3; ++m)
						{
							float hs, hl;
							two_sum(hi[m], lo[m], hs, hl);
							hi[m] = hs;
							lo[m] = hl;
						}
					}
				});
				const int I = a.perm[row0 + i];
				unsigned long long bits[3];
#pragma unroll
				for (int k = 0; k < 3; ++k)
				{
					const double ri = (I >= 0 ? a.b[3 * I + k] : 0.0) - (double(hi[k]) + double(lo[k]));
					rr[0] += ri * ri;
					r64[3 * i + k] = ri;
					bits[k] = (unsigned long long)__double_as_longlong(ri);
				}
				if (!alone)
				{
					st_word(&words[row0 + i], (unsigned)bits[0], (unsigned)(bits[0] >> 32), (unsigned)bits[2], tag);
					st_word(&words[(size_t)a.nrows + row0 + i], (unsigned)bits[1], (unsigned)(bits[1] >> 32),
							(unsigned)(bits[2] >> 32), tag);
				}
			}
			leave_f64<1>(S.L.nCh, rr);
			sums_ready();
			rows_sync();  // every product has used the halo's t and l
			// The halo's residual until the rescale: its three doubles in U.x, U.y, R.x, R.y, U.z, R.z.
			fetch_halo<2>(a, S, words, tag, [&](int i, const ResWord(&v)[2]) {
				U[i].x = __uint_as_float(v[0].a), U[i].y = __uint_as_float(v[0].b);
				R[i].x = __uint_as_float(v[1].a), R[i].y = __uint_as_float(v[1].b);
				U[i].z = __uint_as_float(v[0].c), R[i].z = __uint_as_float(v[1].c);
			});
			scalars_wait();
			continue;
		}
		if (mode == 0)
		{
			// p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = d r.
			const float al = sh.al, be = sh.be, as = sh.as;
			struct Row
			{
				float4 u, r, s, w, q, x;
			};
			auto load = [&](int i, Row& v) {
				v.u = U[i], v.r = R[i], v.s = Sv[i], v.w = W[i];
				if (i < nOwn) v.q = P[i], v.x = X[i];
			};
			auto advance = [&](int i, Row& v) {
				if (i < nOwn)
				{
					v.q.x = __fmaf_rn(be, v.q.x, v.u.x);
					v.q.y = __fmaf_rn(be, v.q.y, v.u.y);
					v.q.z = __fmaf_rn(be, v.q.z, v.u.z);
					v.x.x = __fmaf_rn(as, v.q.x, v.x.x);
					v.x.y = __fmaf_rn(as, v.q.y, v.x.y);
					v.x.z = __fmaf_rn(as, v.q.z, v.x.z);
					P[i] = v.q;
					X[i] = v.x;
				}
				v.s.x = __fmaf_rn(be, v.s.x, v.w.x);
				v.s.y = __fmaf_rn(be, v.s.y, v.w.y);
				v.s.z = __fmaf_rn(be, v.s.z, v.w.z);
				v.r.x = __fmaf_rn(-al, v.s.x, v.r.x);
				v.r.y = __fmaf_rn(-al, v.s.y, v.r.y);
				v.r.z = __fmaf_rn(-al, v.s.z, v.r.z);
				v.u.x = __fmul_rn(v.u.w, v.r.x);
				v.u.y = __fmul_rn(v.r.w, v.r.y);
				v.u.z = __fmul_rn(v.s.w, v.r.z);
				Sv[i] = v.s;
				R[i] = v.r;
				U[i] = v.u;
			};
#pragma unroll 1
			for (int i = tid; i < nLoc; i += 2 * kRowThreads)
			{
				const int i2 = i + kRowThreads;
				Row v, v2;
				load(i, v);
				if (i2 < nLoc) load(i2, v2);
				advance(i, v);
				if (i2 < nLoc) advance(i2, v2);
			}
		}
		else
		{
			// After a refresh (and to start): r = r_true / s, u = d r; x folded, p and s rescaled.
			const double inv = sh.inv;
			const bool start = ph == 2;
			const float ratio = start ? 0.f : sh.ratio;
#pragma unroll 1
			for (int i = tid; i < nLoc; i += kRowThreads)
			{
				const int rs = row_of(S, i);
				const float4 u = U[i], r = R[i], s = Sv[i];
				double t[3];
				if (start)
				{
					const int I = a.perm[rs];
#pragma unroll
					for (int k = 0; k < 3; ++k) t[k] = I >= 0 ? a.b[3 * I + k] : 0.0;
				}
				else if (i < nOwn)
				{
#pragma unroll
					for (int k = 0; k < 3; ++k) t[k] = r64[3 * i + k];
				}
				else
				{
					t[0] = __hiloint2double(__float_as_int(u.y), __float_as_int(u.x));
					t[1] = __hiloint2double(__float_as_int(r.y), __float_as_int(r.x));
					t[2] = __hiloint2double(__float_as_int(r.z), __float_as_int(u.z));
				}
				float rn[3];
#pragma unroll
				for (int k = 0; k < 3; ++k) rn[k] = __double2float_rn(t[k] * inv);
				U[i] = make_float4(__fmul_rn(u.w, rn[0]), __fmul_rn(r.w, rn[1]), __fmul_rn(s.w, rn[2]), u.w);
				R[i] = make_float4(rn[0], rn[1], rn[2], r.w);
				Sv[i] = make_float4(__fmul_rn(s.x, ratio), __fmul_rn(s.y, ratio), __fmul_rn(s.z, ratio), s.w);
				if (i < nOwn && !start)
				{
					const float4 q = P[i], xi = X[i];
					const float xd[3] = {xi.x, xi.y, xi.z};
#pragma unroll
					for (int k = 0; k < 3; ++k)
					{
						float2& xo = a.xhl[3 * (size_t)rs + k];
						float hs, he, h2, l2;
						two_sum(xo.x, xd[k], hs, he);
						two_sum(hs, __fadd_rn(he, xo.y), h2, l2);
						xo = make_float2(h2, l2);
					}
					X[i] = make_float4(0.f, 0.f, 0.f, 0.f);
					P[i] = make_float4(__fmul_rn(q.x, ratio), __fmul_rn(q.y, ratio), __fmul_rn(q.z, ratio), 0.f);
				}
			}
		}
		rows_sync();
		// w of the own rows; r.u, w.u, |r|^2: FP32 over a chunk's rows, pairs over chunks, warps and CTAs.
		ResWord* words = a.rowWords + ((ph & 1) ? (size_t)a.nrows : 0);
		Pair sum[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
		int next = S.head;  // chunks are looked up one ahead
#pragma unroll 1
		for (int j = S.first; j < S.last; ++j)
		{
			const int c = next, i = 32 * c + lane;
			if (j + 1 < S.last) next = a.chunkList[j + 1];
			float w0 = 0.f, w1 = 0.f, w2 = 0.f;
			multiply(S, U, c, w0, w1, w2);
			if (!alone) send_xyz(&words[row0 + i], w0, w1, w2, tag);
			W[i] = make_float4(w0, w1, w2, 0.f);
			const float4 r = R[i], u = U[i];
			float g = 0.f, dl = 0.f, rr = 0.f;
			g += r.x * u.x;
			dl += w0 * u.x;
			rr += r.x * r.x;
			g += r.y * u.y;
			dl += w1 * u.y;
			rr += r.y * r.y;
			g += r.z * u.z;
			dl += w2 * u.z;
			rr += r.z * r.z;
			g = warp_sum(g);
			dl = warp_sum(dl);
			rr = warp_sum(rr);
			sum[0] = sum[0] + Pair{g, 0.f};
			sum[1] = sum[1] + Pair{dl, 0.f};
			sum[2] = sum[2] + Pair{rr, 0.f};
		}
		if (lane == 0)
#pragma unroll
			for (int k = 0; k < 3; ++k) sh.red[k][warp] = make_float2(sum[k].h, sum[k].l);
		sums_ready();
		// Warps without a chunk left wait here for the others: their polls would take the shared-memory pipe from them.
		rows_sync();
		fetch_halo<1>(a, S, words, tag, [&](int i, const ResWord(&v)[1]) { put_xyz(W[i], v[0]); });
		scalars_wait();
	}
	for (int i = tid; i < nOwn; i += kRowThreads)
	{
		const int I = a.perm[row0 + i];
		if (I < 0) continue;
		const float4 xi = X[i];
		const float xd[3] = {xi.x, xi.y, xi.z};
#pragma unroll
		for (int k = 0; k < 3; ++k)
		{
			const float2 x = a.xhl[3 * (size_t)(row0 + i) + k];
			a.x[3 * I + k] = (double(x.x) + double(x.y)) + double(xd[k]);
		}
	}
}

// ---- FP64 -------------------------------------------------------------------------------------------------
// Eigen's conjugate_gradient (Jacobi, zero start, |r|^2 < max(tol^2 |b|^2, DBL_MIN) before the iteration
// is counted, iteration cap). p of the own and the halo rows is advanced in every CTA that uses it, from
// the exchanged z; an iteration has two all-gathers (p.q, then |r|^2 and r.z).
// 1 / r.z, formed while words travel, leaves FP64's range where r.z is below 1e-308 and |r|^2 not yet (right-hand
// sides near 1e-150, a diagonal above one): such systems are solved for kUp times their right-hand side.
constexpr double kUp = 0x1p400, kTinyNorm2 = 1e-150;
template <int kForm, bool kCluster>
__device__ __forceinline__ unsigned talk_f64(const ResArgs& a, const ResPart p, int rhs, unsigned base)
{
	const Talk<kCluster> T = open_talk<kCluster>(a, p, rhs, Types<kForm>::bs);
	const int cap = a.segMaxIter ? a.segMaxIter[p.seg] : a.maxIter;
	unsigned ph = 1;
	double v[2];
	sums_wait();
	total_f64<2>(a, T, ph, base + ph, v, [] {});
	const double bb = v[0];
	double threshold = fmax(a.tol * a.tol * bb, DBL_MIN);
	double rz = v[1], rr = v[0];
	int iter = 0, converged = 1;
	int mode = (bb == 0.0 || bb < threshold || !isfinite(bb)) ? 3 : 0;
	if (!isfinite(bb)) converged = 0;
	if (given_up()) mode = 3;
	const bool tiny = mode == 0 && bb < kTinyNorm2;
	sh.tiny = tiny;
	if (tiny)
	{
		threshold *= kUp * kUp;
		rz *= kUp * kUp;
	}
	publish(mode);
	while (mode != 3)
	{
		++ph;
		beat(a, p, ph);
		sums_wait();
		double pq[1], rzInv = 0.0;
		bool lost = false;  // as in talk_mixed
		total_f64<1>(a, T, ph, base + ph, pq, [&] { lost = given_up(); });
		sh.alpha = rz / pq[0];
		if (lost)
		{
			converged = 0;
			publish(3);
			break;
		}
		publish(0);
		++ph;
		sums_wait();
		total_f64<2>(a, T, ph, base + ph, v, [&] {
			rzInv = 1.0 / rz;
			lost = given_up();
		});
		rr = v[0];
		// rr >= 0 and the threshold compare as integers (no FP64 instruction); NaN and infinity are above.
		const long long bits = __double_as_longlong(rr) & 0x7fffffffffffffffLL;
		sh.beta = v[1] * rzInv;
		if (bits < __double_as_longlong(threshold))
			mode = 3;
		else if (bits >= 0x7ff0000000000000LL)
		{
			converged = 0;  // a NaN residual never converges
			mode = 3;
		}
		else
		{
			rz = v[1];
			iter += 1;
			if (iter >= cap)
			{
				converged = 0;
				mode = 3;
			}
		}
		if (lost) mode = 3;
		publish(mode);
	}
	if (tiny) rr *= 1.0 / (kUp * kUp);
	if (p.rank == 0 && (threadIdx.x & 31) == 0) write_result(a, p, rhs, bb, rr, iter, 0, converged, !isfinite(rr));
	return ph;
}

template <int kForm>
__device__ __forceinline__ void rows_f64(const ResArgs& a, const ResPart part_, int rhs, unsigned base)
{
	// Vectors are walked element by element (bs a row), so a share of a few chunks still spreads its FP64
	// operations over all four schedulers.
	constexpr int bs = Types<kForm>::bs;
	using D = typename Types<kForm>::D;
	const int tid = threadIdx.x;
	const Share S = open_share<kForm>(a, part_);
	const int nOwn = bs * S.L.nOwn, nLoc = bs * S.L.nLoc;
	double* p = shm<double>(S.L.loc);
	double* z = p + nLoc;
	double* x = shm<double>(S.L.own);
	double* r = x + nOwn;
	double* d = r + nOwn;
	double* q = d + nOwn;
	const double* part = shm<double>(S.L.part);
	double* xOut = a.x + (size_t)rhs * a.vecStride;
	ResWord* words = a.rowWords + (size_t)rhs * a.rowStride;  // bs words a row
	const int e0 = 32 * bs * S.c0;
	const bool alone = part_.g == 1;
	unsigned ph = 1;
	rows_sync();

	double v[2] = {0.0, 0.0};
#pragma unroll 1
	for (int e = tid; e < nLoc; e += kRowThreads)
	{
		const int I = a.perm[row_of(S, e / bs)], k = e % bs;
		const double* b = a.b + (size_t)rhs * a.vecStride;
		const D* invdiag = static_cast<const D*>(a.invdiag);
		const double be = I >= 0 ? b[bs * I + k] : 0.0, de = I >= 0 ? double(invdiag[bs * I + k]) : 0.0;
		const double ze = de * be;
		p[e] = ze;
		if (e < nOwn)
		{
			x[e] = 0.0;
			r[e] = be;
			d[e] = de;
			v[0] = fma(be, be, v[0]);
			v[1] = fma(be, ze, v[1]);
		}
	}
	leave_f64<2>(S.L.nCh * bs, v);
	sums_ready();
	rows_sync();
	scalars_wait();
	if (sh.tiny)
	{
		for (int e = tid; e < nLoc; e += kRowThreads)
		{
			p[e] *= kUp;
			if (e < nOwn) r[e] *= kUp;
		}
		rows_sync();
	}
#pragma unroll 1
	while (sh.mode != 3)
	{
		AccMul<kForm> acc{S.L.loc, S.L.own + 3 * 8 * nOwn, S.L.part, {}};
		product<kForm>(S, acc);
		rows_sync();
		double pq[1] = {0.0};
#pragma unroll 1
		for (int e = tid; e < nOwn; e += kRowThreads)
		{
			const int c = e / (32 * bs);
			const int pc = shm<int>(S.L.pieces)[c];
			double t = q[e];
			if (!(pc >> 16))
			{
				const double* y = part + (e - c * (32 * bs));
				t = y[(pc & 255) * (32 * bs)];
#pragma unroll 1
				for (int w = ((pc & 255) >> 1) + 1; w <= pc >> 8; ++w) t += y[w * (64 * bs)];
				q[e] = t;
			}
			pq[0] = fma(p[e], t, pq[0]);
		}
		++ph;
		leave_f64<1>(S.L.nCh * bs, pq);
		sums_ready();
		scalars_wait();
		if (sh.mode == 3) break;
		const double alpha = sh.alpha;
		++ph;
		const unsigned tag = base + ph;
		v[0] = v[1] = 0.0;
#pragma unroll 1
		for (int e = tid; e < nOwn; e += kRowThreads)
		{
			const double re = fma(-alpha, q[e], r[e]);
			const double ze = d[e] * re;
			r[e] = re;
			z[e] = ze;
			if (!alone)
			{
				const unsigned long long u = (unsigned long long)__double_as_longlong(ze);
				st_word(&words[e0 + e], (unsigned)u, (unsigned)(u >> 32), 0u, tag);
			}
			v[0] = fma(re, re, v[0]);
			v[1] = fma(re, ze, v[1]);
		}
		leave_f64<2>(S.L.nCh * bs, v);
		sums_ready();
#pragma unroll 1
		for (int e = tid; e < nOwn; e += kRowThreads) x[e] = fma(alpha, p[e], x[e]);
		fetch_words<bs>(a, S, words, tag, [&](int e, const ResWord& w) {
			z[e] = __longlong_as_double((long long)(((unsigned long long)w.b << 32) | w.a));
		});
		scalars_wait();
		if (sh.mode == 3) break;
		const double beta = sh.beta;
#pragma unroll 1
		for (int e = tid; e < nLoc; e += kRowThreads) p[e] = fma(beta, p[e], z[e]);
		rows_sync();
	}
	for (int e = tid; e < nOwn; e += kRowThreads)
	{
		const int I = a.perm[32 * S.c0 + e / bs];
		if (I >= 0) xOut[(size_t)bs * I + e % bs] = sh.tiny ? x[e] * (1.0 / kUp) : x[e];
	}
}

}  // namespace

// CTAs draw their shares in order, so the shares of a system go to CTAs that come free one after the other and
// at most one system waits for its last shares; every system drawn whole finishes.
template <int kForm, bool kCluster>
__global__ void __launch_bounds__(kResThreads, 1) k_res(ResArgs a)
{
	if (threadIdx.x == 0)
	{
		sh.bad = 0;
		sh.phases = 0;
		if (kCluster)
		{
			for (int k = 0; k < 2; ++k)
				asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(shared_address(&clusterBar[k])) : "memory");
			asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
		}
	}
	__syncthreads();
	if (kCluster) cluster_sync();  // every barrier of the cluster is ready
	const unsigned base = *(volatile unsigned*)&a.ctl->epoch;
	// Each role walks the CTA's shares by itself (what one keeps in registers does not burden the other) and
	// meets the other before each.
	if (threadIdx.x >= kRowThreads)
	{
#pragma unroll 1
		for (;;)
		{
			share_draw();
			const int t = *(volatile int*)&sh.task;
			if (t >= a.nTasks) break;
			const int2 task = a.tasks[t];
			unsigned ph;
			if constexpr (res_mixed(kForm))
				ph = talk_mixed<kCluster>(a, a.parts[task.x], base);
			else
				ph = talk_f64<kForm, kCluster>(a, a.parts[task.x], task.y, base);
			if ((threadIdx.x & 31) == 0) sh.phases = max(sh.phases, ph);
		}
	}
	else
	{
		int round = 0;
#pragma unroll 1
		for (;;)
		{
			// After a wait that gave up every other ends at once, so the shares that are left go by fast.
			// (A cluster's CTAs are one system's in order.)
			if (threadIdx.x == 0)
				sh.task = *(volatile int*)&sh.bad ? a.nTasks : (kCluster ? (int)blockIdx.x + round : (int)atomicAdd(&a.ctl->ticket, 1u));
			round += a.nTasks;
			share_draw();
			const int t = *(volatile int*)&sh.task;
			if (t >= a.nTasks) break;
			const int2 task = a.tasks[t];
			if constexpr (res_mixed(kForm))
				rows_mixed<kForm>(a, a.parts[task.x], base);
			else
				rows_f64<kForm>(a, a.parts[task.x], task.y, base);
			rows_sync();
		}
	}
	__syncthreads();
	if (kCluster)
	{
		cluster_sync();  // no CTA leaves while another may still write to it
		if (*(volatile int*)a.err)  // the same answer in every CTA: whoever gave up did so before the barrier
		{
			if (threadIdx.x >= kRowThreads) settle_cluster();
			__syncthreads();
			cluster_sync();
		}
	}
	// The last CTA to finish moves the tags past those of this launch.
	if (threadIdx.x == 0)
	{
		atomicMax(&a.ctl->maxPhase, sh.phases);
		__threadfence();
		if (atomicAdd(&a.ctl->done, 1u) == gridDim.x - 1)
		{
			__threadfence();
			a.ctl->epoch = base + *(volatile unsigned*)&a.ctl->maxPhase + 1u;
			a.ctl->maxPhase = 0u;
			a.ctl->ticket = 0u;
			a.ctl->done = 0u;
		}
	}
}

namespace {
using ResKernel = void (*)(ResArgs);
ResKernel res_kernel(int form, bool cluster)
{
	switch (form)
	{
	case kResF64: return cluster ? k_res<kResF64, true> : k_res<kResF64, false>;
	case kResF64M: return k_res<kResF64M, false>;
	case kResF64S: return cluster ? k_res<kResF64S, true> : k_res<kResF64S, false>;
	case kResMixedFar: return k_res<kResMixedFar, false>;
	default: return cluster ? k_res<kResMixed, true> : k_res<kResMixed, false>;
	}
}
}  // namespace

cudaError_t res_set_max_dynamic_smem(int form, int bytes)
{
	const cudaError_t e = cudaFuncSetAttribute(res_kernel(form, false), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
	if (e != cudaSuccess || res_kernel(form, true) == res_kernel(form, false)) return e;
	return cudaFuncSetAttribute(res_kernel(form, true), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

bool res_cluster_fits(int form, int ctas, size_t smem)
{
	const ResKernel kernel = res_kernel(form, true);
	if (ctas < 2 || ctas > kResCluster || kernel == res_kernel(form, false)) return false;
	if (ctas > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
	{
		cudaGetLastError();
		return false;
	}
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(ctas);
	cfg.blockDim = dim3(kResThreads);
	cfg.dynamicSmemBytes = smem;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim = {(unsigned)ctas, 1, 1};
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	int n = 0;
	if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess) return n > 0;
	cudaGetLastError();
	return false;
}

cudaError_t res_launch(int form, int grid, size_t smem, const ResArgs& a, cudaStream_t s)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(kResThreads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cudaLaunchAttribute attr[1];
	if (a.cluster)
	{
		attr[0].id = cudaLaunchAttributeClusterDimension;
		attr[0].val.clusterDim = {(unsigned)grid, 1, 1};
	}
	else
	{
		attr[0].id = cudaLaunchAttributeCooperative;  // the CTAs of a system wait for one another
		attr[0].val.cooperative = 1;
	}
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, res_kernel(form, a.cluster), a);
}

}  // namespace gbfem
