// hex8_gl.cuh -- geometrically nonlinear (total Lagrangian, Green-Lagrange
// strain) HEX8 element, the NONLINEAR_STRAIN branch of
// StructuralElement3D::internal_residual (src/elasticity/solid_element_3d.cpp:
// 299-409, strain operator initialize_green_lagrange_strain_operator :1309-1463)
// with the isotropic St Venant-Kirchhoff material of
// IsotropicMaterialProperty::StiffnessMatrix3D
// (src/property_cards/isotropic_material_property_card.cpp:512-528).
//
// Written per node pair instead of with the reference's 6 x 24 strain
// operators.  With Fd = I + grad u (rows f_i) and physical shape gradients g_a,
// the strain variation of dof (component i, node a) is sym(f_i (x) g_a), so
//   internal force   f_ia = sum_qp JxW (Fd S g_a)_i
//   material tangent K_ia,jb = sum_qp JxW [lam (f_i.g_a)(f_j.g_b)
//                                  + mu ((f_i.f_j)(g_a.g_b) + (f_i.g_b)(f_j.g_a))]
//   geometric        + delta_ij sum_qp JxW g_a.S.g_b
// with S = lam tr(E) I + 2 mu E, E = (Fd^T Fd - I)/2 (the second Piola-Kirchhoff
// stress of C applied to the Green-Lagrange strain in Voigt form).
//
// With the sums T = sum_qp JxW (Fd g_a) (x) (Fd g_b) and s = sum_qp JxW g_a.S.g_b, the block
// of nodes a, b is lam T + mu T^T + mu sum_qp JxW (g_a.g_b) Fd Fd^T + s I: 21 products per
// Gauss point instead of 41 with the terms scaled inside the sum, and the block of b, a is
// its transpose.
//
// The work is split into items ((point), (point, node), (dof), (node pair)) over the
// element's workspace; the items of a phase only read what earlier phases wrote, so a
// kernel may spread them over any threads with a barrier between phases.  The phase_*
// functions do the items of one lane of a warp per element (the host tests run the same
// source as a loop over 32 lanes).
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define GL_HD __host__ __device__ __forceinline__
#else
#define GL_HD inline
#endif

namespace mg {
namespace gl {

// workspace of the linear-strain element (doubles; 488 = 3.9 KB)
struct LinearWork {
    double X[24], w[8], inv[8][9], g[8][8][3];
    double wg[8][8][3];  // JxW (times the point's modulus, if it has one) g_a
};

// element workspace (doubles; 1,064 = 8.5 KB)
struct Work {
    double X[24];         // node coordinates, node-major (3 a + d)
    double u[24];         // displacements, node-major (3 a + c)
    double w[8];          // JxW per Gauss point (unit weights)
    double inv[8][9];     // inverse Jacobian per Gauss point
    double g[8][8][3];    // physical gradients g[q][a]
    double Fd[8][9];      // deformation gradient I + grad u per Gauss point
    double wS[8][6];      // JxW times the second Piola-Kirchhoff stress: xx, yy, zz, xy, yz, zx
    double wB[8][6];      // JxW Fd Fd^T (f_i . f_j), in the same order
    double Fg[8][8][3];   // Fd g_a  (f_i . g_a)
    double wFg[8][8][3];  // JxW Fd g_a
    double wSg[8][8][3];  // JxW S g_a
};

// reference gradient of shape function a at Gauss point q = i + 2 j + 4 k
// (libMesh HEX8 node order: x signs - + + -, y signs - - + +, z - for nodes 0-3).
// Each component is +-1/2 times the other two directions' hats, each (1 + 1/sqrt 3) / 2 at
// the node's own side and (1 - 1/sqrt 3) / 2 at the other: one of three constants.
GL_HD void dref(int q, int a, double d[3]) {
    constexpr double near = 0.5 * (1.0 + 0.57735026918962576451), far = 0.5 * (1.0 - 0.57735026918962576451);
    constexpr double c0 = 0.5 * far * far, c1 = 0.5 * near * far, c2 = 0.5 * near * near;
    const int ax = (a + 1) >> 1 & 1, ay = a >> 1 & 1, az = a >> 2 & 1;
    const int mx = (q & 1) == ax, my = (q >> 1 & 1) == ay, mz = (q >> 2 & 1) == az;
    const double x = my & mz ? c2 : my | mz ? c1 : c0;
    const double y = mx & mz ? c2 : mx | mz ? c1 : c0;
    const double z = mx & my ? c2 : mx | my ? c1 : c0;
    d[0] = ax ? x : -x;
    d[1] = ay ? y : -y;
    d[2] = az ? z : -z;
}

// item (q): Jacobian, JxW, inverse into s.inv[at], s.w[at].  Returns false for a
// non-positive determinant.  (W: any workspace with X, w, inv.)
template <class W>
GL_HD bool jacobian_at(W &s, int q, int at) {
    double J[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // J[i][j] = d x_j / d xi_i
    for (int a = 0; a < 8; a++) {
        double d[3];
        dref(q, a, d);
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) J[i * 3 + j] += d[i] * s.X[a * 3 + j];
    }
    double iv[9];
    iv[0] = J[4] * J[8] - J[5] * J[7];
    iv[1] = J[2] * J[7] - J[1] * J[8];
    iv[2] = J[1] * J[5] - J[2] * J[4];
    iv[3] = J[5] * J[6] - J[3] * J[8];
    iv[4] = J[0] * J[8] - J[2] * J[6];
    iv[5] = J[2] * J[3] - J[0] * J[5];
    iv[6] = J[3] * J[7] - J[4] * J[6];
    iv[7] = J[1] * J[6] - J[0] * J[7];
    iv[8] = J[0] * J[4] - J[1] * J[3];
    const double det = J[0] * iv[0] + J[1] * iv[3] + J[2] * iv[6];
    const double r = 1.0 / det;
    for (int k = 0; k < 9; k++) s.inv[at][k] = iv[k] * r;
    s.w[at] = det;
    return det > 0.0;
}
template <class W>
GL_HD bool jacobian_item(W &s, int q) {
    return jacobian_at(s, q, q);
}

// item (q, a): physical gradient g_j = sum_k (d xi_k / d x_j) d phi / d xi_k
template <class W>
GL_HD void gradient_item(W &s, int q, int a) {
    double d[3];
    dref(q, a, d);
    const double *iv = s.inv[q];
    for (int j = 0; j < 3; j++) s.g[q][a][j] = iv[j * 3] * d[0] + iv[j * 3 + 1] * d[1] + iv[j * 3 + 2] * d[2];
}

// item (q): Fd, Green-Lagrange strain, JxW S, JxW Fd Fd^T.  The strain is formed from
// H = grad u as (H + H^T + H^T H) / 2, not as (Fd^T Fd - I) / 2, whose subtraction would
// cancel the leading digits of small strains (a 1e-8 strain would keep only 8 significant
// digits).
GL_HD void stress_item(Work &s, int q, double lam, double mu) {
    double H[9], Fd[9];
    for (int i = 0; i < 9; i++) H[i] = 0.0;
    for (int a = 0; a < 8; a++)
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) H[i * 3 + j] += s.u[a * 3 + i] * s.g[q][a][j];
    for (int i = 0; i < 9; i++) {
        Fd[i] = H[i] + (i % 4 == 0 ? 1.0 : 0.0);
        s.Fd[q][i] = Fd[i];
    }
    const double w = s.w[q];
    double E[6];  // xx, yy, zz, xy, yz, zx
    for (int r = 0; r < 6; r++) {
        const int j = r % 3, k = r < 3 ? j : (j + 1) % 3;
        double c = 0.0;
        for (int m = 0; m < 3; m++) c += H[m * 3 + j] * H[m * 3 + k];
        E[r] = 0.5 * (H[j * 3 + k] + H[k * 3 + j] + c);
        double b = 0.0;
        for (int m = 0; m < 3; m++) b += Fd[j * 3 + m] * Fd[k * 3 + m];
        s.wB[q][r] = w * b;
    }
    const double ltr = lam * (E[0] + E[1] + E[2]);
    for (int r = 0; r < 6; r++) s.wS[q][r] = w * (2.0 * mu * E[r] + (r < 3 ? ltr : 0.0));
}

// item (q, a): Fd g_a, JxW Fd g_a and JxW S g_a
GL_HD void projection_item(Work &s, int q, int a) {
    const double g[3] = {s.g[q][a][0], s.g[q][a][1], s.g[q][a][2]};
    const double w = s.w[q];
    const double *S = s.wS[q];
    for (int i = 0; i < 3; i++) {
        const double f = s.Fd[q][i * 3] * g[0] + s.Fd[q][i * 3 + 1] * g[1] + s.Fd[q][i * 3 + 2] * g[2];
        s.Fg[q][a][i] = f;
        s.wFg[q][a][i] = w * f;
    }
    s.wSg[q][a][0] = S[0] * g[0] + S[3] * g[1] + S[5] * g[2];
    s.wSg[q][a][1] = S[3] * g[0] + S[1] * g[1] + S[4] * g[2];
    s.wSg[q][a][2] = S[5] * g[0] + S[4] * g[1] + S[2] * g[2];
}

// item (a, i): internal force of dof (i, a)
GL_HD double force_item(const Work &s, int a, int i) {
    double f = 0.0;
    for (int q = 0; q < 8; q++) {
        const double *Fd = s.Fd[q] + i * 3;
        const double *Sg = s.wSg[q][a];
        f += Fd[0] * Sg[0] + Fd[1] * Sg[1] + Fd[2] * Sg[2];
    }
    return f;
}

// item (node pair (a, b)): the 3 x 3 tangent block K[i][j] = K_ia,jb
GL_HD void phase_tangent(const Work &s, int a, int b, double lam, double mu, double K[9]) {
    double T[9], B[6], sg = 0.0;
    for (int k = 0; k < 9; k++) T[k] = 0.0;
    for (int k = 0; k < 6; k++) B[k] = 0.0;
#ifdef __CUDA_ARCH__
#pragma unroll 2
#endif
    for (int q = 0; q < 8; q++) {
        const double *ga = s.g[q][a], *gb = s.g[q][b], *Sb = s.wSg[q][b];
        const double *Fa = s.wFg[q][a], *Fb = s.Fg[q][b], *wB = s.wB[q];
        const double gab = ga[0] * gb[0] + ga[1] * gb[1] + ga[2] * gb[2];
        sg += ga[0] * Sb[0] + ga[1] * Sb[1] + ga[2] * Sb[2];
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) T[i * 3 + j] += Fa[i] * Fb[j];
        for (int r = 0; r < 6; r++) B[r] += gab * wB[r];
    }
    for (int i = 0; i < 3; i++) {
        K[i * 4] = (lam + mu) * T[i * 4] + (mu * B[i] + sg);
        const int j = (i + 1) % 3;
        const double m = mu * B[3 + i];
        K[i * 3 + j] = lam * T[i * 3 + j] + (mu * T[j * 3 + i] + m);
        K[j * 3 + i] = lam * T[j * 3 + i] + (mu * T[i * 3 + j] + m);
    }
}

// item (node pair (a, b)) of the linear element: lam T + mu T^T + mu tr(T) I with
// T = sum_qp JxW g_a (x) g_b
GL_HD void linear_pair_item(const LinearWork &s, int a, int b, double lam, double mu, double K[9]) {
    double T[9];
    for (int k = 0; k < 9; k++) T[k] = 0.0;
    for (int q = 0; q < 8; q++) {
        const double *ga = s.wg[q][a], *gb = s.g[q][b];
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) T[i * 3 + j] += ga[i] * gb[j];
    }
    const double mtr = mu * (T[0] + T[4] + T[8]);
    for (int i = 0; i < 3; i++) {
        K[i * 4] = (lam + mu) * T[i * 4] + mtr;
        const int j = (i + 1) % 3;
        K[i * 3 + j] = lam * T[i * 3 + j] + mu * T[j * 3 + i];
        K[j * 3 + i] = lam * T[j * 3 + i] + mu * T[i * 3 + j];
    }
}

// the items of lane `lane` of a warp that evaluates one element (workspaces with X, u)
template <class W>
GL_HD bool phase_jacobian(W &s, int lane) {
    return lane >= 8 || jacobian_item(s, lane);
}
template <class W>
GL_HD void phase_gradients(W &s, int lane) {
    for (int p = lane; p < 64; p += 32) gradient_item(s, p >> 3, p & 7);
}
GL_HD void phase_stress(Work &s, int lane, double lam, double mu) {
    if (lane < 8) stress_item(s, lane, lam, mu);
}
GL_HD void phase_projections(Work &s, int lane) {
    for (int p = lane; p < 64; p += 32) projection_item(s, p >> 3, p & 7);
}
GL_HD double phase_force(const Work &s, int lane) { return force_item(s, lane / 3, lane % 3); }

// ---------------------------------------------------------------------------
// Stress output (StructuralElement3D::calculate_stress, solid_element_3d.cpp:
// 1147-1270; von Mises and its derivatives, stress_output_base.cpp:183-271;
// the KS weights of ks_stress_output.cpp:41-99).  Per Gauss point: the strain
// (linear: B u; nonlinear: the Green-Lagrange strain), sigma = C eps with the
// stress modulus, sigma_vm, ex = exp(p (sigma_vm - s0) / s0), and the tensor T
// of t = C (d sigma_vm / d sigma) (T_jj = t_j, off-diagonal = the shear entry),
// so that d sigma_vm / d u_ia = (Fd T g_a)_i with Fd = I (linear) or I + grad u.
// ---------------------------------------------------------------------------
struct StressWork {
    double X[24], u[24], w[8], inv[8][9], g[8][8][3];
    double Fd[8][9];
    double T[8][9];
    double vm[8];
    double ex[8];
};

// lanes 0-7, q = lane
GL_HD void phase_von_mises(StressWork &s, int lane, double lam, double mu, bool nonlinear,
                           double p_ks, double sigma0) {
    if (lane >= 8) return;
    const int q = lane;
    double H[9];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double v = 0.0;
            for (int a = 0; a < 8; a++) v += s.u[a * 3 + i] * s.g[q][a][j];
            H[i * 3 + j] = v;
            s.Fd[q][i * 3 + j] = (nonlinear ? v : 0.0) + (i == j ? 1.0 : 0.0);
        }
    // Voigt strain [xx, yy, zz, xy, yz, zx], engineering shears
    static constexpr int VJ[6] = {0, 1, 2, 0, 1, 0}, VK[6] = {0, 1, 2, 1, 2, 2};
    double eps[6];
    for (int r = 0; r < 6; r++) {
        const int j = VJ[r], k = VK[r];
        double e = (r < 3) ? H[j * 3 + j] : H[j * 3 + k] + H[k * 3 + j];
        if (nonlinear) {
            double c = 0.0;
            for (int m = 0; m < 3; m++) c += H[m * 3 + j] * H[m * 3 + k];
            e += (r < 3) ? 0.5 * c : c;
        }
        eps[r] = e;
    }
    const double tr = eps[0] + eps[1] + eps[2];
    double sg[6];
    for (int r = 0; r < 3; r++) sg[r] = lam * tr + 2.0 * mu * eps[r];
    for (int r = 3; r < 6; r++) sg[r] = mu * eps[r];
    const double P = 0.5 * ((sg[0] - sg[1]) * (sg[0] - sg[1]) + (sg[1] - sg[2]) * (sg[1] - sg[2]) +
                            (sg[2] - sg[0]) * (sg[2] - sg[0])) +
                     3.0 * (sg[3] * sg[3] + sg[4] * sg[4] + sg[5] * sg[5]);
    const double vm = sqrt(P);
    double d[6] = {0, 0, 0, 0, 0, 0};  // d sigma_vm / d sigma, zero where sigma_vm = 0
    if (P > 0.0) {
        const double c = 0.5 / vm;
        d[0] = c * (2.0 * sg[0] - sg[1] - sg[2]);
        d[1] = c * (2.0 * sg[1] - sg[2] - sg[0]);
        d[2] = c * (2.0 * sg[2] - sg[0] - sg[1]);
        for (int r = 3; r < 6; r++) d[r] = c * 6.0 * sg[r];
    }
    const double trd = d[0] + d[1] + d[2];
    double *T = s.T[q];
    T[0] = lam * trd + 2.0 * mu * d[0];
    T[4] = lam * trd + 2.0 * mu * d[1];
    T[8] = lam * trd + 2.0 * mu * d[2];
    T[1] = T[3] = mu * d[3];
    T[5] = T[7] = mu * d[4];
    T[2] = T[6] = mu * d[5];
    s.vm[q] = vm;
    s.ex[q] = exp(p_ks * (vm - sigma0) / sigma0);
}

// lanes 0-23, lane = 3 a + i: sum_qp ex JxW d sigma_vm / d u_ia
GL_HD double phase_vm_gradient(const StressWork &s, int lane) {
    const int a = lane / 3, i = lane % 3;
    double acc = 0.0;
    for (int q = 0; q < 8; q++) {
        const double *g = s.g[q][a], *T = s.T[q], *F = s.Fd[q] + i * 3;
        double Tg[3];
        for (int m = 0; m < 3; m++) Tg[m] = T[m * 3] * g[0] + T[m * 3 + 1] * g[1] + T[m * 3 + 2] * g[2];
        acc += s.w[q] * s.ex[q] * (F[0] * Tg[0] + F[1] * Tg[1] + F[2] * Tg[2]);
    }
    return acc;
}

}  // namespace gl
}  // namespace mg
