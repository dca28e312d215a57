// The host side of the C entry points (gbfem_host.cpp, gbfem_plan.cpp) on a stand-in for the CUDA runtime that
// lives in host memory: two devices, allocations that can be made to fail, solves that can be made to report that
// a wait ran out. Kernels do nothing. Runs the case named on the command line and prints "ok" or what went wrong.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <limits>
#include <map>
#include <new>
#include <random>
#include <string>
#include <vector>

#include "../../include/gbfem.h"
#include "gbfem_internal.h"
#include "gbfem_pcg.h"
#include "gbfem_plan.h"
#include "gbfem_res.h"

#define CHECK(x)                                              \
	do                                                        \
		if (!(x))                                             \
		{                                                     \
			std::printf("line %d: %s\n", __LINE__, #x);       \
			std::exit(1);                                     \
		}                                                     \
	while (0)

long long fake_int32_max = 2147483647;  // INT32_MAX of the sources under test

// ---- the stand-in -------------------------------------------------------------------------------------------------
namespace fake {

int device = 0;                          // current device
std::map<std::pair<int, int>, int> res;  // dynamic shared memory limit of a resident form on a device
std::map<std::pair<int, int>, int> pcg;  // and of a persistent one
std::map<void*, size_t> blocks;          // device memory
long long allocations = 0, failAt = -1;  // the allocation that fails, counted from zero
long long news = 0, newFails = -1;       // the same of the host's memory, which `new` gives
int solves = 0;
bool giveUp = false;                     // whether solves report a wait that ran out
bool capturing = false;
std::function<void()> solve;             // repeated by a graph launch

int limit(const std::map<std::pair<int, int>, int>& m, int form)
{
	const auto it = m.find({device, form});
	return it == m.end() ? 48 * 1024 : it->second;
}

}  // namespace fake

void* operator new(size_t n)
{
	if (fake::news++ == fake::newFails) throw std::bad_alloc();
	if (void* p = std::malloc(n ? n : 1)) return p;
	throw std::bad_alloc();
}
void* operator new(size_t n, const std::nothrow_t&) noexcept { return std::malloc(n ? n : 1); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {

cudaError_t cudaGetDevice(int* d)
{
	*d = fake::device;
	return cudaSuccess;
}
cudaError_t cudaSetDevice(int d)
{
	if (d < 0 || d > 1) return cudaErrorInvalidDevice;
	fake::device = d;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
	*v = a == cudaDevAttrMultiProcessorCount ? 152 : (a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 228 * 1024 : 0);
	return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n)
{
	if (fake::allocations++ == fake::failAt) return cudaErrorMemoryAllocation;
	*p = std::calloc(n, 1);
	const long long fails = fake::newFails, news = fake::news;
	fake::newFails = -1;  // the record below is not the caller's
	fake::blocks[*p] = n;
	fake::newFails = fails;
	fake::news = news;
	return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
	CHECK(fake::blocks.erase(p) == 1);
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
	*p = std::calloc(n, 1);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
	CHECK(n == 0 || (d && s));
	if (n && !fake::capturing) std::memmove(d, s, n);
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
	return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t)
{
	CHECK(n == 0 || d);
	if (n && !fake::capturing) std::memset(d, v, n);
	return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
	fake::capturing = true;
	return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*)
{
	fake::capturing = false;
	return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long)
{
	*e = reinterpret_cast<cudaGraphExec_t>(&fake::solve);
	return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t)
{
	fake::solve();
	return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }

}  // extern "C"

namespace gbfem {

cudaError_t res_set_max_dynamic_smem(int form, int bytes)
{
	fake::res[{fake::device, form}] = bytes;
	return cudaSuccess;
}
bool res_cluster_fits(int, int, size_t) { return false; }
cudaError_t res_launch(int form, int, size_t smem, const ResArgs& a, cudaStream_t)
{
	if ((long long)smem > fake::limit(fake::res, form)) return cudaErrorInvalidValue;
	CHECK(a.parts && a.tasks && a.lcol && a.off && a.perm && a.ctl && a.seg && a.err && a.b && a.x && a.val && a.invdiag);
	CHECK(a.mail && a.rowWords);
	if (res_mixed(form)) CHECK(a.xhl && a.r64 && a.chunkWarp && a.chunkList);
	auto run = [a] {
		CHECK(*a.err == 0);  // a flag left set would end this launch's waits at once
		++fake::solves;
		for (int t = 0; t < a.nTasks; ++t)
		{
			SegCtl& c = a.seg[a.parts[a.tasks[t].x].seg + (size_t)a.tasks[t].y * a.segStride];
			c = SegCtl{};
			c.bb = 1.0;
			c.converged = 1;
			c.iter = 3;
		}
		if (fake::giveUp) *a.err = 1;
	};
	if (!fake::capturing) run();
	if (fake::capturing) fake::solve = run;
	return cudaSuccess;
}
cudaError_t pcg_set_max_dynamic_smem(int form, int bytes)
{
	fake::pcg[{fake::device, form}] = bytes;
	return cudaSuccess;
}
cudaError_t pcg_occupancy(int, int* n, size_t)
{
	*n = 4;
	return cudaSuccess;
}
cudaError_t pcg_launch(int form, const cudaLaunchConfig_t& cfg, const PcgArgs& a)
{
	if ((long long)cfg.dynamicSmemBytes > fake::limit(fake::pcg, form)) return cudaErrorInvalidValue;
	for (int s = 0; s < a.nsegs && !fake::capturing; ++s) a.seg[s].converged = 1;
	++fake::solves;
	return cudaSuccess;
}
void launch_step_accumulate(const SegCtl*, int nseg, const int*, const int* err, double* acc, cudaStream_t)
{
	fake::solve = [=, before = fake::solve] {
		before();
		if (*err) acc[4 * nseg + 1] = 1.0;
	};
}

void launch_mcg_init(int, int, const double* B, const uint8_t*, const double*, const float*, double*, double*, double*,
					 double*, McgCtl* ctl, double* part, double, int, const Launch&)
{
	CHECK(B && ctl && part);
	ctl->allDone = 1;
	for (int& c : ctl->converged) c = 1;
}
void launch_node_rotation(const DevBody&, const double* Qe, double* Wn, cudaStream_t) { CHECK(Qe && Wn); }
void launch_element_adjoint(const DevBody&, const double*, const double*, const double* mu, const double* dv, double, double,
							double, double* gx, double* gv, double*, double*, cudaStream_t, bool)
{
	CHECK(mu && dv && gx && gv);
}
void launch_scatter_values(int, const int* idx, const double* v, double*, cudaStream_t) { CHECK(idx && v); }
void launch_state_update(int, const double*, double* dvPrev, const double* xt, double*, double*, double, int newton, CgCtl*,
						 double*, const Launch&)
{
	CHECK(xt && (!newton || dvPrev));
}
void launch_assemble_full_csc(int, const int* a, const int* b, const int* c, const int* d, const double* k, const double* m,
							  const uint8_t*, double, double, double* S, cudaStream_t)
{
	CHECK(a && b && c && d && k && m && S);
}

}  // namespace gbfem

// ---- the cases ----------------------------------------------------------------------------------------------------
namespace {

// a x b x c unit cubes of six tetrahedra, the first node fixed, `spare` nodes of no element after the others.
struct Grid
{
	std::vector<double> X, Ey, Nu, Rho;
	std::vector<int32_t> T, bc{0, 1, 2};
	gbfem_mesh_desc desc{};
	Grid(int a, int b, int c, int spare = 0, double at = 0.0)
	{
		auto id = [&](int i, int j, int k) { return (i * (b + 1) + j) * (c + 1) + k; };
		for (int i = 0; i <= a; ++i)
			for (int j = 0; j <= b; ++j)
				for (int k = 0; k <= c; ++k)
					for (double v : {0.01 * i, 0.01 * j, 0.01 * k}) X.push_back(v);
		X.insert(X.end(), 3 * spare, at);
		const int order[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
		for (int i = 0; i < a; ++i)
			for (int j = 0; j < b; ++j)
				for (int k = 0; k < c; ++k)
					for (int o = 0; o < 6; ++o)
					{
						int p[3] = {i, j, k};
						int t[4] = {id(p[0], p[1], p[2])};
						for (int s = 0; s < 3; ++s)
						{
							++p[order[o][s]];
							t[s + 1] = id(p[0], p[1], p[2]);
						}
						if (o == 1 || o == 2 || o == 5) std::swap(t[2], t[3]);  // odd orders: a positive volume
						T.insert(T.end(), t, t + 4);
					}
		const size_t E = T.size() / 4;
		Ey.assign(E, 1e5);
		Nu.assign(E, 0.4);
		Rho.assign(E, 1000.0);
		desc = gbfem_mesh_desc{(int32_t)(X.size() / 3), X.data(), (int32_t)E, T.data(), Ey.data(), Nu.data(), Rho.data(),
							   (int32_t)bc.size(), bc.data()};
	}
};

gbfem_params params(int precision, int device)
{
	gbfem_params p;
	gbfem_params_default(&p);
	p.precision = precision;
	p.device = device;
	return p;
}

gbfem_handle create(const Grid& g, int precision, int device = 0)
{
	const gbfem_params p = params(precision, device);
	gbfem_handle h = nullptr;
	CHECK(gbfem_create(&g.desc, &p, &h) == GBFEM_OK);
	return h;
}

// Bodies, compliance and caller's matrices on a second device after the same on the first.
void two_devices()
{
	const Grid g(10, 10, 10);
	for (int precision : {GBFEM_PRECISION_FP64, GBFEM_PRECISION_MIXED})
		for (int device = 0; device < 2; ++device)
		{
			gbfem_handle h = create(g, precision, device);
			CHECK(gbfem_step(h, 1e-3, 1, 0) == GBFEM_OK);
			std::vector<double> b(3 * g.X.size(), 1.0), x(b.size());
			CHECK(gbfem_apply_compliance(h, 3, b.data(), x.data(), 0, nullptr) == GBFEM_OK);
			gbfem_destroy(h);
		}
	const int n = 4000;
	std::vector<int32_t> ptr{0}, row;
	std::vector<double> val;
	for (int c = 0; c < n; ++c)
	{
		row.push_back(c);
		val.push_back(4.0);
		if (c + 1 < n) row.push_back(c + 1), val.push_back(-1.0);
		ptr.push_back((int32_t)row.size());
	}
	for (int device = 0; device < 2; ++device)
	{
		gbfem_cg cg = nullptr;
		CHECK(gbfem_cg_create(n, ptr.data(), row.data(), val.data(), device, &cg) == GBFEM_OK);
		std::vector<double> b(n, 1.0), x(n);
		CHECK(gbfem_cg_solve(cg, b.data(), x.data(), nullptr, nullptr) == GBFEM_OK);
		gbfem_cg_destroy(cg);
	}
}

// f() with each of its allocations failing in turn, and again once memory is there; then without a failure.
template <typename F>
void every_allocation(F f)
{
	for (int k = 0;; ++k)
	{
		fake::failAt = fake::allocations + k;
		const gbfem_status st = f();
		const bool failed = fake::allocations > fake::failAt;
		fake::failAt = -1;
		if (!failed)
		{
			CHECK(st == GBFEM_OK);
			return;
		}
		CHECK(st == GBFEM_OUT_OF_MEMORY);
		if (k % 2 == 0) continue;  // two failures in a row as well as one
		CHECK(f() == GBFEM_OK);
	}
}

// Calls whose buffers cannot be had report it and can be made again.
void failed_allocations()
{
	const Grid g(6, 6, 6);
	const size_t n = g.X.size();
	std::vector<double> b(200 * n, 1.0), x(200 * n), y(n), z(n), w(n);
	std::vector<int32_t> dofs(n);
	for (int precision : {GBFEM_PRECISION_FP64, GBFEM_PRECISION_MIXED})
	{
		gbfem_params p = params(precision, 0);
		p.newton_max_iterations = 2;
		gbfem_handle h = nullptr;
		every_allocation([&] {
			if (h) gbfem_destroy(h);
			h = nullptr;
			return gbfem_create(&g.desc, &p, &h);
		});
		every_allocation([&] { return gbfem_step(h, 1e-3, 1, precision == GBFEM_PRECISION_FP64 ? GBFEM_STEP_KEEP_SYSTEM : 0); });
		for (int columns : {3, 200, 3, 40})
			every_allocation([&] {
				return gbfem_apply_compliance(h, columns, b.data(), x.data(), GBFEM_COMPLIANCE_WARPING, nullptr);
			});
		every_allocation([&] { return gbfem_set_velocities(h, 1, dofs.data(), b.data()); });
		every_allocation([&] { return gbfem_set_velocities(h, (int)n, dofs.data(), b.data()); });
		every_allocation([&] {
			return gbfem_adjoint_step(h, 1e-3, b.data(), b.data(), b.data(), b.data(), b.data(), y.data(), z.data(), w.data(),
									  nullptr, 0);
		});
		gbfem_destroy(h);
		// A batch: columns eight at a time; rollouts.
		const gbfem_mesh_desc two[2] = {g.desc, g.desc};
		p.newton_max_iterations = 1;
		CHECK(gbfem_batch_create(2, two, &p, &h) == GBFEM_OK);
		CHECK(gbfem_step(h, 1e-3, 1, 0) == GBFEM_OK);
		std::vector<double> lx(2 * n), lv(2 * n), x0(2 * n), v0(2 * n);
		every_allocation([&] {
			return gbfem_apply_compliance(h, 2, b.data(), x.data(), GBFEM_COMPLIANCE_WARPING, nullptr);
		});
		for (int steps : {2, 6})
		{
			every_allocation([&] {
				return gbfem_rollout_forward(h, 1e-3, steps, steps / 2, b.data(), b.data(), x0.data(), v0.data());
			});
			every_allocation([&] {
				return gbfem_rollout_backward(h, b.data(), b.data(), lx.data(), lv.data(), nullptr, nullptr);
			});
		}
		gbfem_destroy(h);
	}
	gbfem_cg cg = nullptr;
	const std::vector<int32_t> ptr{0, 1, 2}, row{0, 1};
	every_allocation([&] {
		if (cg) gbfem_cg_destroy(cg);
		cg = nullptr;
		return gbfem_cg_create(2, ptr.data(), row.data(), b.data(), 0, &cg);
	});
	gbfem_cg_destroy(cg);
}

// Compliance calls that run out of host memory say so.
void failed_host_memory()
{
	const Grid g(6, 6, 6);
	const size_t n = g.X.size();
	const gbfem_params p = params(GBFEM_PRECISION_FP64, 0);
	const gbfem_mesh_desc two[2] = {g.desc, g.desc};
	std::vector<double> b(80 * n, 1.0), x(80 * n);
	for (int batch = 0; batch < 2; ++batch)
	{
		gbfem_handle h = nullptr;
		CHECK((batch ? gbfem_batch_create(2, two, &p, &h) : gbfem_create(&g.desc, &p, &h)) == GBFEM_OK);
		CHECK(gbfem_step(h, 1e-3, 1, 0) == GBFEM_OK);
		for (int columns : {2, 40})
			for (int k = 0;; ++k)
			{
				fake::newFails = fake::news + k;
				const gbfem_status st = gbfem_apply_compliance(h, columns, b.data(), x.data(), 0, nullptr);
				const bool failed = fake::news > fake::newFails;
				fake::newFails = -1;
				CHECK(st == (failed ? GBFEM_OUT_OF_MEMORY : GBFEM_OK));
				if (!failed) break;
			}
		gbfem_destroy(h);
	}
}

// A solve that gives up is reported by its own call; the next one starts with a clear flag (res_launch looks).
void errors_reported_once()
{
	const Grid g(6, 6, 6);
	const size_t n = g.X.size();
	std::vector<double> b(3 * n, 1.0), x(3 * n), y(n), z(n), w(n);
	gbfem_handle h = nullptr;
	auto once = [&](auto f) {
		fake::giveUp = true;
		CHECK(f() == GBFEM_CUDA_ERROR);
		fake::giveUp = false;
		const int before = fake::solves;
		CHECK(gbfem_step(h, 1e-3, 1, 0) == GBFEM_OK && fake::solves > before);
		CHECK(f() == GBFEM_OK);
	};
	for (int precision : {GBFEM_PRECISION_FP64, GBFEM_PRECISION_MIXED})
	{
		const bool mixed = precision == GBFEM_PRECISION_MIXED;
		gbfem_params p = params(precision, 0);
		p.autotune = mixed;
		CHECK(gbfem_create(&g.desc, &p, &h) == GBFEM_OK);
		once([&] { return gbfem_step(h, 1e-3, 1, 0); });  // mixed: in the autotuner
		if (mixed) CHECK(gbfem_set_tuning(h, 64, 4, 2, GBFEM_CG_ONE_PHASE) == GBFEM_OK);
		once([&] { return gbfem_step(h, 1e-3, 1, 0); });
		once([&] { return gbfem_apply_compliance(h, 3, b.data(), x.data(), 0, nullptr); });
		once([&] {
			return gbfem_adjoint_step(h, 1e-3, b.data(), b.data(), b.data(), b.data(), b.data(), y.data(), z.data(), w.data(),
									  nullptr, 0);
		});
		if (mixed)
		{
			once([&] { return gbfem_step(h, 1e-3, 1, GBFEM_STEP_GRAPH); });
			once([&] { return gbfem_rollout_forward(h, 1e-3, 4, 2, b.data(), b.data(), y.data(), z.data()); });
			once([&] { return gbfem_rollout_backward(h, b.data(), b.data(), y.data(), z.data(), nullptr, nullptr); });
		}
		gbfem_destroy(h);
	}
}

// Nodes of no element at NaN and at infinity: orders stay permutations that keep the others in theirs, and a body
// with such nodes is created as before.
void positions_without_an_order()
{
	const double nan = std::numeric_limits<double>::quiet_NaN(), inf = std::numeric_limits<double>::infinity();
	std::mt19937 rng(1);
	for (int trial = 0; trial < 60; ++trial)
	{
		const int n = 33 + (int)(rng() % 3000), every = 1 + trial % 7;
		std::vector<double> X(3 * n);
		for (double& v : X) v = rng() % every == 0 ? (rng() % 4 == 0 ? inf : nan) : rng() * 1e-9;
		const std::vector<int> w(n, 5);
		std::vector<int> seen(n, 0);
		for (int i : gbfem::res_chunk_order(X, w)) ++seen.at(i);
		for (const auto& part : gbfem::res_node_parts(X.data(), w, 1 + n / 200))
			for (int i : part) ++seen.at(i);
		for (int s : seen) CHECK(s == 2);
		CHECK((int)gbfem::res_curve_keys(X.data(), n).size() == n);
	}
	for (int trial = 0; trial < 20; ++trial)
	{
		// Along a line, two parts: every number of the first lies before every one of the second.
		const int n = 640;
		std::vector<double> X(3 * n, 0.0);
		for (int i = 0; i < n; ++i) X[3 * i] = rng() % 4 == 0 ? nan : rng() * 1e-9;
		const auto parts = gbfem::res_node_parts(X.data(), std::vector<int>(n, 1), 2);
		double last = -inf, first = inf;
		for (int i : parts[0]) last = std::fmax(last, X[3 * i]);
		for (int i : parts[1]) first = std::fmin(first, X[3 * i]);
		CHECK(parts.size() == 2 && last <= first);
	}
	for (int precision : {GBFEM_PRECISION_FP64, GBFEM_PRECISION_MIXED})
		for (double at : {nan, inf}) gbfem_destroy(create(Grid(9, 9, 9, 700, at), precision));
}

// A wait runs out by the clock, but not at the end of a pause in which nothing ran; progress elsewhere begins it again.
void patience()
{
	const long long limit = 1000000000, poll = 1000;
	unsigned long long t = 12345;
	auto polls = [&](gbfem::ResPatience& p, unsigned beat, long long most) {  // until it has run out, at most `most`
		long long n = 0;
		for (; n < most; ++n)
		{
			t += poll;
			if (p.look() && p.over(t, beat, limit)) break;
		}
		return n;
	};
	gbfem::ResPatience p;
	CHECK(polls(p, 7, 1000) == 1000);
	t += 5 * limit;  // the GPU runs another program for five seconds
	CHECK(polls(p, 7, 1000) == 1000);
	CHECK(polls(p, 8, 1000) == 1000);  // some system advances
	CHECK(polls(p, 8, limit / poll - 1000) == limit / poll - 1000);
	const long long end = polls(p, 8, limit);
	CHECK(end < 1300);  // the limit after the look that saw the advance
	gbfem::ResPatience q;  // pauses alone
	for (int k = 0; k < 2000; ++k, t += limit) CHECK(polls(q, 0, 1) == 1);
	CHECK(polls(q, 0, limit) < 300);
}

// The order of the rows does not decide what is accepted: an FP64 batch, whose rows go into compact shares of about ten
// chunks, needs no larger range of indices than a mixed one in node order.
void index_range()
{
	std::vector<Grid> grids;
	for (int k = 0; k < 70; ++k) grids.emplace_back(5, 6 + k % 3, 7);
	std::vector<gbfem_mesh_desc> meshes;
	for (const Grid& g : grids) meshes.push_back(g.desc);
	auto accepted = [&](int precision) {
		const gbfem_params p = params(precision, 0);
		gbfem_handle h = nullptr;
		const gbfem_status st = gbfem_batch_create((int)meshes.size(), meshes.data(), &p, &h);
		if (h) gbfem_destroy(h);
		return st == GBFEM_OK;
	};
	long long lo = 2000000, hi = 10000000;  // refused, accepted
	while (hi - lo > 30000)
	{
		fake_int32_max = (lo + hi) / 2;
		(accepted(GBFEM_PRECISION_MIXED) ? hi : lo) = fake_int32_max;
	}
	fake_int32_max = hi;
	CHECK(lo > 2000000 && hi < 10000000);
	CHECK(accepted(GBFEM_PRECISION_FP64));
	fake_int32_max = lo;
	CHECK(!accepted(GBFEM_PRECISION_FP64));
}

}  // namespace

int main(int argc, char** argv)
{
	const std::map<std::string, void (*)()> cases = {
		{"two_devices", two_devices},
		{"failed_allocations", failed_allocations},
		{"failed_host_memory", failed_host_memory},
		{"errors_reported_once", errors_reported_once},
		{"positions_without_an_order", positions_without_an_order},
		{"patience", patience},
		{"index_range", index_range},
	};
	const auto it = cases.find(argc > 1 ? argv[1] : "");
	CHECK(it != cases.end());
	it->second();
	CHECK(fake::blocks.empty());
	std::printf("ok\n");
	return 0;
}
