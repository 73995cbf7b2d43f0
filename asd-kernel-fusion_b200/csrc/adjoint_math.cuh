// adjoint_math.cuh -- vector helpers and the vector-Jacobian product of the LLG
// right-hand side, shared by the two adjoints (adjoint.cu, adjoint_resident.cu).
// Included after llg_math.cuh inside an anonymous namespace of each file.
#pragma once

__device__ __forceinline__ V3 v3(double x, double y, double z) { return V3{x, y, z}; }
__device__ __forceinline__ V3 vadd(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 vsub(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ V3 vmul(double s, V3 a) { return v3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ double vdot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 vcross(V3 a, V3 b) {
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

constexpr int NPAR = 6;  // J1, J2, alpha, hx, hy, hz

// The vector-Jacobian product of f at stage state sv for the adjoint m of one
// (site, replica), with the sums nn and nnn of sv's nearest and diagonal
// neighbours: P = S x nu (to be gathered by the neighbours), the local part l,
// and the parameter derivatives added to part[] (formulas: adjoint.cu).
__device__ __forceinline__ void vjp_vals(const LLGArgs &a, const V3 &sv, const V3 &nn,
                                         const V3 &nnn, const V3 &m, V3 &p, V3 &l,
                                         double (&part)[NPAR]) {
    const V3 H = vadd(vadd(vmul(a.J1, nn), vmul(a.J2, nnn)), v3(a.hx, a.hy, a.hz));
    const V3 tau = vcross(H, sv);
    const V3 nu = vmul(a.g, vadd(m, vmul(a.alpha, vcross(m, sv))));
    p = vcross(sv, nu);
    l = vadd(vmul(a.g * a.alpha, vcross(tau, m)), vcross(nu, H));
    const V3 sxt = vcross(sv, tau);
    const V3 f = vmul(a.g, vadd(tau, vmul(a.alpha, sxt)));
    part[0] += vdot(p, nn);
    part[1] += vdot(p, nnn);
    part[2] += vdot(m, vadd(vmul(-2.0 * a.alpha * a.g, f), vmul(a.g, sxt)));
    part[3] += p.x;
    part[4] += p.y;
    part[5] += p.z;
}
