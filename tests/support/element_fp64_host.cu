// Test support only: the FP64 form's element (gbfem_element_fp64.cuh) and the general one
// (gbfem_element.cuh), compiled for the host, on the same inputs.
#include <cmath>

#include "gbfem_element_fp64.cuh"

namespace {
struct Out
{
	double* K;    // 4 x 4 blocks of 9, [4 a + b], a >= b
	double* rhs;
	bool blocks() const { return true; }
	void rhs_entry(int a, int i, double v) { rhs[3 * a + i] = v; }
	void block(int a, int b, const double (&blk)[9])
	{
		for (int k = 0; k < 9; ++k) K[9 * (4 * a + b) + k] = blk[k];
	}
};
}  // namespace

// x, x0, uK, uM: 4 nodes of 3 in ascending order; g: 4 shape-function gradients of 3. K and rhs (general: the
// same layout, every block). Returns the general flags + 8 times the FP64 form's.
extern "C" int gbfem_host_element_fp64(const double* x, const double* x0, const double* uK, const double* uM,
									   const double* g, double lamV, double muV, double cm, int lumped, double* K,
									   double* rhs, double* Kgen, double* rhsGen)
{
	gbfem::elem::ElemIn in;
	double G[4][3], p[3][3], q[3][3], uk[3][3], um[4][3], g3[3][3], kfull[144], ks[90], fdbg[12];
	for (int a = 0; a < 4; ++a)
	{
		in.nd[a] = a;
		for (int k = 0; k < 3; ++k)
		{
			in.p[a][k] = x[3 * a + k] - x[k];
			in.q[a][k] = x0[3 * a + k] - x0[k];
			in.uK[a][k] = uK[3 * a + k];
			in.uM[a][k] = um[a][k] = uM[3 * a + k];
			in.vv[a][k] = 0.0;
			G[a][k] = g[3 * a + k];
			if (a == 0) continue;
			p[a - 1][k] = in.p[a][k];
			q[a - 1][k] = in.q[a][k];
			uk[a - 1][k] = uK[3 * a + k] - uK[k];
			g3[a - 1][k] = g[3 * a + k];
		}
	}
	in.alphaDbg = in.betaDbg = 0.0;
	in.lumped = lumped;
	const int fl = gbfem::elem::compute<double, true>(in, G, lamV, muV, cm, ks, 1, rhsGen, 1, kfull, fdbg);
	for (int a = 0; a < 4; ++a)
		for (int b = 0; b < 4; ++b)
			for (int i = 0; i < 3; ++i)
				for (int j = 0; j < 3; ++j) Kgen[9 * (4 * a + b) + 3 * i + j] = kfull[(3 * a + i) * 12 + 3 * b + j];
	Out out{K, rhs};
	return fl + 8 * gbfem::elem::compute_fp64(p, q, uk, um, g3, lamV, muV, cm, lumped != 0, out);
}
