// gbfem_element_fp64.cuh -- the corotational tetrahedron of the FP64 form: the element of
// gbfem_element.cuh (compute_to) arranged for the fewest FP64 instructions.
//
// An FP64 instruction takes a scheduler 64 cycles here, against 2 in FP32, and nothing else the element
// kernel does comes near: its time is its count of FP64 instructions. Against compute_to this form
//   - works in the rotated frame: with V = F R^T (symmetric), H = (tr V I - V)^-1, h_a = R g_a and
//     wr_c = x_c - x_0 - R (x0_c - x0_0), the terms of compute_to become
//       T'_a [g_b x r_q]_q = N_a [h_b]x,   N_a = (lambda h_a zeta^T + mu [rows: h_a x W_i]
//                                                + [mu sum_c G_ac wr_c - R y_a]x) H,
//     with no product by R per node and block (R G^-1 = R H R^T R drops out of both sides);
//   - forms node 0 from the others (the gradients, and with them h, N, y and the forces, sum to zero) and
//     takes every displacement relative to it;
//   - takes the rotation from FP32 Newton steps, refined in FP64 to FP64 accuracy (rotation_fp64);
//   - has the nodes in ascending order, so the stored lower blocks are the same for all elements of a
//     warp (in mesh order a warp ran through both triangles).
#pragma once

#include <cmath>

#include "gbfem_element.cuh"

namespace gbfem {
namespace elem {

// R (row-major) of F = R S and flag 1 for the SVD path, as rotation() gives. The FP32 polar factor is about
// 1e-7 off; as a unit quaternion it is orthogonal to FP64 accuracy. For R off by exp([w]x), F R^T is off
// symmetry by [a]x with a = (tr V I - V) w + O(w^2), so w = H a with H in FP32 is off by 1e-7 |w| and
// |w|^2: two such steps reach FP64 accuracy. Elements that FP32 calls near-degenerate, and those whose
// second step is not small, take the FP64 path.
__host__ __device__ __forceinline__ int rotation_fp64(const double (&F)[9], double (&R)[9])
{
	float f[9], r[9];
#pragma unroll
	for (int k = 0; k < 9; ++k) f[k] = float(F[k]);
	if (polar_newton(f, r))
	{
		float q[4];
		const float t = r[0] + r[4] + r[8];
		if (t > 0.f)
		{
			q[0] = 1.f + t;
			q[1] = r[7] - r[5];
			q[2] = r[2] - r[6];
			q[3] = r[3] - r[1];
		}
		else if (r[0] > r[4] && r[0] > r[8])
		{
			q[0] = r[7] - r[5];
			q[1] = 1.f + r[0] - r[4] - r[8];
			q[2] = r[1] + r[3];
			q[3] = r[2] + r[6];
		}
		else if (r[4] > r[8])
		{
			q[0] = r[2] - r[6];
			q[1] = r[1] + r[3];
			q[2] = 1.f + r[4] - r[0] - r[8];
			q[3] = r[5] + r[7];
		}
		else
		{
			q[0] = r[3] - r[1];
			q[1] = r[2] + r[6];
			q[2] = r[5] + r[7];
			q[3] = 1.f + r[8] - r[0] - r[4];
		}
		const float qi = 1.f / sqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
		double Q[4];
#pragma unroll
		for (int k = 0; k < 4; ++k) Q[k] = double(q[k] * qi);
		// H = (tr V I - V)^-1 with V = F R^T, all in FP32.
		float H[9];
		{
			const float v01 = 0.5f * (f[0] * r[3] + f[1] * r[4] + f[2] * r[5] + f[3] * r[0] + f[4] * r[1] + f[5] * r[2]);
			const float v02 = 0.5f * (f[0] * r[6] + f[1] * r[7] + f[2] * r[8] + f[6] * r[0] + f[7] * r[1] + f[8] * r[2]);
			const float v12 = 0.5f * (f[3] * r[6] + f[4] * r[7] + f[5] * r[8] + f[6] * r[3] + f[7] * r[4] + f[8] * r[5]);
			const float v00 = f[0] * r[0] + f[1] * r[1] + f[2] * r[2], v11 = f[3] * r[3] + f[4] * r[4] + f[5] * r[5],
						v22 = f[6] * r[6] + f[7] * r[7] + f[8] * r[8];
			const float A[9] = {v11 + v22, -v01, -v02, -v01, v00 + v22, -v12, -v02, -v12, v00 + v11};
			cofactor3(A, H);
			const float id = 1.f / (A[0] * H[0] + A[1] * H[1] + A[2] * H[2]);
#pragma unroll
			for (int k = 0; k < 9; ++k) H[k] *= id;
		}
		float w[3];
#pragma unroll
		for (int step = 0; step < 2; ++step)
		{
			// Unit length: |Q|^2 = 1 + d with d ~ 1e-7, then 1e-13.
			const double d = Q[0] * Q[0] - 1.0 + Q[1] * Q[1] + Q[2] * Q[2] + Q[3] * Q[3];
			const double s = step == 0 ? 1.0 + d * (-0.5 + 0.375 * d) : 1.0 - 0.5 * d;
#pragma unroll
			for (int k = 0; k < 4; ++k) Q[k] *= s;
			const double x2 = 2.0 * Q[1], y2 = 2.0 * Q[2], z2 = 2.0 * Q[3];
			const double wx = Q[0] * x2, wy = Q[0] * y2, wz = Q[0] * z2, xx = 1.0 - Q[1] * x2, yy = Q[2] * y2;
			R[0] = 1.0 - yy - Q[3] * z2;
			R[1] = Q[1] * y2 - wz;
			R[2] = Q[1] * z2 + wy;
			R[3] = Q[1] * y2 + wz;
			R[4] = xx - Q[3] * z2;
			R[5] = Q[2] * z2 - wx;
			R[6] = Q[1] * z2 - wy;
			R[7] = Q[2] * z2 + wx;
			R[8] = xx - yy;
			const float a0 = float(F[6] * R[3] - F[3] * R[6] + F[7] * R[4] - F[4] * R[7] + F[8] * R[5] - F[5] * R[8]);
			const float a1 = float(F[0] * R[6] - F[6] * R[0] + F[1] * R[7] - F[7] * R[1] + F[2] * R[8] - F[8] * R[2]);
			const float a2 = float(F[3] * R[0] - F[0] * R[3] + F[4] * R[1] - F[1] * R[4] + F[5] * R[2] - F[2] * R[5]);
#pragma unroll
			for (int i = 0; i < 3; ++i) w[i] = H[3 * i] * a0 + H[3 * i + 1] * a1 + H[3 * i + 2] * a2;
			if (step == 0)
			{
				// Q <- (1, w / 2) Q
				const double u[3] = {double(0.5f * w[0]), double(0.5f * w[1]), double(0.5f * w[2])};
				const double p[4] = {Q[0], Q[1], Q[2], Q[3]};
				Q[0] = p[0] - u[0] * p[1] - u[1] * p[2] - u[2] * p[3];
				Q[1] = p[1] + u[0] * p[0] + u[1] * p[3] - u[2] * p[2];
				Q[2] = p[2] + u[1] * p[0] + u[2] * p[1] - u[0] * p[3];
				Q[3] = p[3] + u[2] * p[0] + u[0] * p[2] - u[1] * p[1];
			}
		}
		if (w[0] * w[0] + w[1] * w[1] + w[2] * w[2] <= 1e-18f)
		{
			// R <- R + [w]x R: |w| is at most 1e-9, and its square at rounding.
			const double u[3] = {double(w[0]), double(w[1]), double(w[2])};
#pragma unroll
			for (int j = 0; j < 3; ++j)
			{
				const double c0 = R[j], c1 = R[3 + j], c2 = R[6 + j];
				R[j] = c0 + u[1] * c2 - u[2] * c1;
				R[3 + j] = c1 + u[2] * c0 - u[0] * c2;
				R[6 + j] = c2 + u[0] * c1 - u[1] * c0;
			}
			return 0;
		}
	}
	if (polar_newton(F, R)) return 0;
	polar_svd(F, R);
	return 1;
}

// D = sum_c u_c h_c^T over nodes 1..3 (u_0 = 0).
__host__ __device__ __forceinline__ void outer3(const double (&u)[3][3], const double (&h)[4][3], double (&D)[3][3])
{
#pragma unroll
	for (int i = 0; i < 3; ++i)
#pragma unroll
		for (int j = 0; j < 3; ++j) D[i][j] = u[0][i] * h[1][j] + u[1][i] * h[2][j] + u[2][i] * h[3][j];
}

// (Krot u)_a of nodes 1..3 for u_0 = 0 and D = sum_c u_c h_c^T: lambda tr(D) h_a + mu D^T h_a + mu sum_c G_ac u_c.
__host__ __device__ __forceinline__ void krot_apply(const double (&u)[3][3], const double (&D)[3][3], const double (&h)[4][3],
													const double (&muG)[4][4], double lamV, double muV, double (&out)[3][3])
{
	const double tr = lamV * (D[0][0] + D[1][1] + D[2][2]);
	double E[3][3];
#pragma unroll
	for (int j = 0; j < 3; ++j)
#pragma unroll
		for (int i = 0; i < 3; ++i) E[j][i] = i == j ? muV * D[i][j] + tr : muV * D[i][j];
#pragma unroll
	for (int a = 0; a < 3; ++a)
#pragma unroll
		for (int j = 0; j < 3; ++j)
			out[a][j] = E[j][0] * h[a + 1][0] + E[j][1] * h[a + 1][1] + E[j][2] * h[a + 1][2] + muG[a + 1][1] * u[0][j] +
						muG[a + 1][2] * u[1][j] + muG[a + 1][3] * u[2][j];
}

// The element's results as compute_to defines them, for nodes 0..3 in ascending order of their ids; p, q, uK of
// nodes 1..3 relative to node 0, g of nodes 1..3. Out: block(a, b, blk) for a >= b, rhs_entry(a, i, v).
// kPart: the whole element (-1), or a quarter of its results: the right-hand side (0), the blocks of node 3 (1), of
// node 2 (2), of nodes 0 and 1 (3).
template <int kPart = -1, typename Out>
__host__ __device__ __forceinline__ int compute_fp64(const double (&p)[3][3], const double (&q)[3][3],
													 const double (&uK)[3][3], const double (&uM)[4][3],
													 const double (&g)[3][3], double lamV, double muV, double cm, bool lumped,
													 Out& out)
{
	double F[9], R[9];
#pragma unroll
	for (int i = 0; i < 3; ++i)
#pragma unroll
		for (int j = 0; j < 3; ++j) F[3 * i + j] = p[0][i] * g[0][j] + p[1][i] * g[1][j] + p[2][i] * g[2][j];
	int flags = rotation_fp64(F, R);
	// H = (tr V I - V)^-1 (symmetric); det of compute_to's G is that of tr V I - V.
	double H[9];
	bool extra;
	{
		const double v00 = F[0] * R[0] + F[1] * R[1] + F[2] * R[2], v11 = F[3] * R[3] + F[4] * R[4] + F[5] * R[5],
					 v22 = F[6] * R[6] + F[7] * R[7] + F[8] * R[8];
		const double m01 = F[0] * R[3] + F[1] * R[4] + F[2] * R[5], m02 = F[0] * R[6] + F[1] * R[7] + F[2] * R[8],
					 m12 = F[3] * R[6] + F[4] * R[7] + F[5] * R[8];
		const double a = v11 + v22, b = v00 + v22, c = v00 + v11;  // the off-diagonal entries are -m
		const double c00 = b * c - m12 * m12, c11 = a * c - m02 * m02, c22 = a * b - m01 * m01;
		const double c01 = m02 * m12 + m01 * c, c02 = m01 * m12 + m02 * b, c12 = m01 * m02 + m12 * a;
		const double d = a * c00 - m01 * c01 - m02 * c02;
		extra = fabs(d) > 1e-12;
		const double id = 1.0 / d;
		H[0] = c00 * id;
		H[4] = c11 * id;
		H[8] = c22 * id;
		H[1] = H[3] = c01 * id;
		H[2] = H[6] = c02 * id;
		H[5] = H[7] = c12 * id;
		if (!extra) flags |= 2;
	}
	double h[4][3], muG[4][4], w[3][3], wr[3][3];
#pragma unroll
	for (int a = 0; a < 3; ++a)
#pragma unroll
		for (int i = 0; i < 3; ++i)
		{
			h[a + 1][i] = R[3 * i] * g[a][0] + R[3 * i + 1] * g[a][1] + R[3 * i + 2] * g[a][2];
			wr[a][i] = p[a][i] - (R[3 * i] * q[a][0] + R[3 * i + 1] * q[a][1] + R[3 * i + 2] * q[a][2]);
		}
#pragma unroll
	for (int i = 0; i < 3; ++i) h[0][i] = -(h[1][i] + h[2][i] + h[3][i]);
#pragma unroll
	for (int a = 1; a < 4; ++a)
#pragma unroll
		for (int c = a; c < 4; ++c)
			muG[a][c] = muG[c][a] = muV * (g[a - 1][0] * g[c - 1][0] + g[a - 1][1] * g[c - 1][1] + g[a - 1][2] * g[c - 1][2]);
#pragma unroll
	for (int a = 1; a < 4; ++a) muG[0][a] = muG[a][0] = -(muG[1][a] + muG[2][a] + muG[3][a]);
	muG[0][0] = -(muG[0][1] + muG[0][2] + muG[0][3]);
	// Ry_a = R (Krot w)_a with w = R^T wr (KTimesRx_x0), nodes 1..3.
	double Ry[3][3], D[3][3];
	{
		double y[3][3];
#pragma unroll
		for (int c = 0; c < 3; ++c)
#pragma unroll
			for (int i = 0; i < 3; ++i) w[c][i] = R[i] * wr[c][0] + R[3 + i] * wr[c][1] + R[6 + i] * wr[c][2];
		outer3(w, h, D);
		krot_apply(w, D, h, muG, lamV, muV, y);
#pragma unroll
		for (int a = 0; a < 3; ++a)
#pragma unroll
			for (int i = 0; i < 3; ++i) Ry[a][i] = R[3 * i] * y[a][0] + R[3 * i + 1] * y[a][1] + R[3 * i + 2] * y[a][2];
	}
	// zeta = sum_c h_c x wr_c and W = sum_c h_c wr_c^T, scaled by the moduli.
	double lz[3], mW[3][3];
	outer3(wr, h, D);
	lz[0] = lamV * (D[2][1] - D[1][2]);
	lz[1] = lamV * (D[0][2] - D[2][0]);
	lz[2] = lamV * (D[1][0] - D[0][1]);
#pragma unroll
	for (int i = 0; i < 3; ++i)
#pragma unroll
		for (int j = 0; j < 3; ++j) mW[i][j] = muV * D[j][i];
	double N[4][9];
#pragma unroll
	for (int a = 0; a < 3; ++a)
	{
		if ((kPart == 1 && a != 2) || (kPart == 2 && a != 1)) continue;
		const double* ha = h[a + 1];
		double t[3], L[9];
#pragma unroll
		for (int k = 0; k < 3; ++k)
			t[k] = muG[a + 1][1] * wr[0][k] + muG[a + 1][2] * wr[1][k] + muG[a + 1][3] * wr[2][k] - Ry[a][k];
#pragma unroll
		for (int i = 0; i < 3; ++i)
		{
			L[3 * i] = ha[i] * lz[0] + ha[1] * mW[i][2] - ha[2] * mW[i][1];
			L[3 * i + 1] = ha[i] * lz[1] + ha[2] * mW[i][0] - ha[0] * mW[i][2];
			L[3 * i + 2] = ha[i] * lz[2] + ha[0] * mW[i][1] - ha[1] * mW[i][0];
		}
		L[1] -= t[2];
		L[2] += t[1];
		L[3] += t[2];
		L[5] -= t[0];
		L[6] -= t[1];
		L[7] += t[0];
#pragma unroll
		for (int i = 0; i < 3; ++i)
#pragma unroll
			for (int j = 0; j < 3; ++j)
				N[a + 1][3 * i + j] = extra ? L[3 * i] * H[j] + L[3 * i + 1] * H[3 + j] + L[3 * i + 2] * H[6 + j] : 0.0;
	}
	if constexpr (kPart != 1 && kPart != 2)
#pragma unroll
		for (int k = 0; k < 9; ++k) N[0][k] = -(N[1][k] + N[2][k] + N[3][k]);
	// Right-hand side: Krot u~ + N zt with u~ = uK - wr, zt = sum_c h_c x u~_c, and the mass term.
	if constexpr (kPart <= 0)
	{
		double ut[3][3], f[3][3], sum[3];
#pragma unroll
		for (int c = 0; c < 3; ++c)
#pragma unroll
			for (int i = 0; i < 3; ++i) ut[c][i] = uK[c][i] - wr[c][i];
		outer3(ut, h, D);
		const double zt[3] = {D[2][1] - D[1][2], D[0][2] - D[2][0], D[1][0] - D[0][1]};
		krot_apply(ut, D, h, muG, lamV, muV, f);
#pragma unroll
		for (int a = 0; a < 3; ++a)
#pragma unroll
			for (int i = 0; i < 3; ++i)
				f[a][i] += N[a + 1][3 * i] * zt[0] + N[a + 1][3 * i + 1] * zt[1] + N[a + 1][3 * i + 2] * zt[2];
		const double own = lumped ? 5.0 * cm : cm;
#pragma unroll
		for (int i = 0; i < 3; ++i)
		{
			sum[i] = lumped ? 0.0 : cm * (uM[0][i] + uM[1][i] + uM[2][i] + uM[3][i]);
			out.rhs_entry(0, i, own * uM[0][i] + (sum[i] - (f[0][i] + f[1][i] + f[2][i])));
		}
#pragma unroll
		for (int a = 0; a < 3; ++a)
#pragma unroll
			for (int i = 0; i < 3; ++i) out.rhs_entry(a + 1, i, own * uM[a + 1][i] + (sum[i] + f[a][i]));
	}
	if (kPart == 0 || !out.blocks()) return flags;
#pragma unroll
	for (int a = 0; a < 4; ++a)
	{
		if ((kPart == 1 && a != 3) || (kPart == 2 && a != 2) || (kPart == 3 && a > 1)) continue;
		const double la[3] = {lamV * h[a][0], lamV * h[a][1], lamV * h[a][2]};
		const double ma[3] = {muV * h[a][0], muV * h[a][1], muV * h[a][2]};
#pragma unroll
		for (int b = 0; b <= a; ++b)
		{
			const double* hb = h[b];
			double blk[9];
#pragma unroll
			for (int i = 0; i < 3; ++i)
			{
				const double* n = N[a] + 3 * i;
				blk[3 * i] = la[i] * hb[0] + ma[0] * hb[i] + n[1] * hb[2] - n[2] * hb[1];
				blk[3 * i + 1] = la[i] * hb[1] + ma[1] * hb[i] + n[2] * hb[0] - n[0] * hb[2];
				blk[3 * i + 2] = la[i] * hb[2] + ma[2] * hb[i] + n[0] * hb[1] - n[1] * hb[0];
				blk[4 * i] += muG[a][b];
			}
			out.block(a, b, blk);
		}
	}
	return flags;
}

}  // namespace elem
}  // namespace gbfem
