// Double-precision kernels of the Lagrange-leapfrog step.
//
// This header is compiled twice:
//   fp64_fast.cu   LULESH_VARIANT=fp64,  LULESH_EXACT=0, FMA contraction on
//   fp64_exact.cu  LULESH_VARIANT=fp64x, LULESH_EXACT=1, nvcc --fmad=false
// With the reference's operand order kept in step_math.cuh, the exact
// variant rounds every operation as the reference does and matches the CPU
// oracle bit for bit (the oracle then uses the same portable cube root). The
// fast variant works in block fixed point on the integer pipes
// (block_fixed.cuh, eos_fixed.cuh), with double forms beside it for what does
// not fit.
//
// One cycle = four phases, each a per-element (or per-node) device function
// used both by the single-problem kernels below and by the batched
// persistent kernels of batch_kernels.cuh:
//   forces_elem      stress + FB hourglass corner forces   (lulesh.cc:787-1113)
//   nodes_node       CSR gather, a = f/m, symmetry BC, v, x (lulesh.cc:838-862, 1115-1158, 566-588)
//   kinematics_elem  volume, arealg, vdov, v <- vnew, Q gradients (lulesh.cc:1169-1418)
//   material_elem    Q limiter, EOS x rep, sound speed, save, dt constraints
//                    (lulesh.cc:1420-1974)
#pragma once

#include "block_fixed.cuh"
#include "step_math.cuh"

namespace lulesh {
namespace LULESH_VARIANT {

#if LULESH_EXACT
// Stress and hourglass corner forces of element i, stored separately
// (corner-major) so that the node gather adds them in the reference's order
// (lulesh.cc:849-856).
__device__ __forceinline__ void forces_elem(const Mesh& m, int i) {
    const size_t N = (size_t)m.numElem;
    int nl[8];
    load_nodelist(m.nodelist, i, nl);
    double x[8], y[8], z[8];
    gather8(m.x, nl, x);
    gather8(m.y, nl, y);
    gather8(m.z, nl, z);

    // stress (InitIntegrateStressForElemsTask, lulesh.cc:787-836)
    {
        const double sig = -LD(m.p + i) - LD(m.q + i);
        if (jacobian_singular(x, y, z)) raise_error(m.result, i, PHASE_FORCES);
        double nx[8], ny[8], nz[8];
        node_normals(nx, ny, nz, x, y, z);          // 16 x the normals
        const double sigs = sig * kInvNormalScale;  // a power of two: exact
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            m.fsx[k * N + i] = -(sigs * nx[k]);
            m.fsy[k * N + i] = -(sigs * ny[k]);
            m.fsz[k * N + i] = -(sigs * nz[k]);
        }
    }

    // hourglass (CalcHourglassForElemsTask, lulesh.cc:864-1113)
    const double determ = LD(m.volo + i) * LD(m.v + i);
    if (determ <= 0.0) {
        raise_error(m.result, i, PHASE_FORCES);
        return;
    }
    double hg[8][4];
    {
        double dvdx[8], dvdy[8], dvdz[8];
        volume_derivs(dvdx, dvdy, dvdz, x, y, z);
        hourgam_all(hg, x, y, z, dvdx, dvdy, dvdz, rcp(determ));
    }
    const double coefficient =
        -m.prm.hgcoef * 0.01 * LD(m.ss + i) * LD(m.elemMass + i) / cbrt_portable(determ);
    double vel[8], f[8];
    double* outs[3] = {m.fhx, m.fhy, m.fhz};
    const double* vels[3] = {m.xd, m.yd, m.zd};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        gather8(vels[a], nl, vel);
        fb_force_axis(hg, vel, coefficient, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) outs[a][k * N + i] = f[k];
    }
}
#else
// Corner forces of element i in double: the path of the elements that do not
// fit the block fixed point of forces_elem (coordinates, velocities or
// scalars that are infinite, NaN or of extreme magnitude, a centre Jacobian
// determinant near zero). Stress plus hourglass, summed in registers and
// stored once (corner-major fsx, fsy, fsz). The zero test on the centre
// Jacobian's determinant (lulesh.cc:817-821) is taken in another summation
// order: zero for the same collapsed elements, though a near-singular element
// may round differently. The hourglass vectors come from the volume gradient
// (192 x dV/dx_k) and the mode sums scaled by volinv / 192. The stress force
// (p + q) n enters through the face vectors scaled by (p + q) / 8 and starts
// each corner's hourglass multiply-add chain. Elements that fail a test store
// nothing: the step reports the error and its state is not used. Bit a of
// `axes`: form and store the forces along axis a.
__device__ __noinline__ void forces_double(const Mesh& m, int i, int axes) {
    const size_t N = (size_t)m.numElem;
    int nl[8];
    load_nodelist(m.nodelist, i, nl);
    double J[3][3], c[3][3], h[3][4], fa[6][3];
    {
        double x[8], y[8], z[8];
        gather8(m.x, nl, x);
        gather8(m.y, nl, y);
        gather8(m.z, nl, z);
        walsh7(x, J[0], h[0]);
        walsh7(y, J[1], h[1]);
        walsh7(z, J[2], h[2]);
        cofactors(J, c);
        face_txs<0, 1, 2, 3>(x, y, z, fa[0]);
        face_txs<0, 4, 5, 1>(x, y, z, fa[1]);
        face_txs<1, 5, 6, 2>(x, y, z, fa[2]);
        face_txs<2, 6, 7, 3>(x, y, z, fa[3]);
        face_txs<3, 7, 4, 0>(x, y, z, fa[4]);
        face_txs<4, 7, 6, 5>(x, y, z, fa[5]);
    }
    if (f_is_zero(J[0][0] * c[0][0] + J[1][0] * c[1][0] + J[2][0] * c[2][0])) raise_error(m.result, i, PHASE_FORCES);
    const double determ = LD(m.volo + i) * LD(m.v + i);
    if (f_le(determ, 0.0)) {
        raise_error(m.result, i, PHASE_FORCES);
        return;
    }
    double hg[8][4];
    {
        double gx[8], gy[8], gz[8];
        volume_gradient(J, c, h[0], h[1], h[2], gx, gy, gz);
        const double sc = rcp(determ) * (1.0 / 192.0);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int a = 0; a < 3; ++a) h[a][k] = pmul(h[a][k], sc);
        hourgam_mode_h<0>(hg, h[0][0], h[1][0], h[2][0], gx, gy, gz);
        hourgam_mode_h<1>(hg, h[0][1], h[1][1], h[2][1], gx, gy, gz);
        hourgam_mode_h<2>(hg, h[0][2], h[1][2], h[2][2], gx, gy, gz);
        hourgam_mode_h<3>(hg, h[0][3], h[1][3], h[2][3], gx, gy, gz);
    }
    const double scale = (LD(m.p + i) + LD(m.q + i)) * kInvNormalScale;
#pragma unroll
    for (int f = 0; f < 6; ++f)
#pragma unroll
        for (int d = 0; d < 3; ++d) fa[f][d] = pmul(fa[f][d], scale);
    const double coefficient = -m.prm.hgcoef * 0.01 * LD(m.ss + i) * LD(m.elemMass + i) * rcbrt_pos(determ);
    double* outs[3] = {m.fsx, m.fsy, m.fsz};
    const double* vels[3] = {m.xd, m.yd, m.zd};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!(axes >> a & 1)) continue;
        double st[8], vel[8], f[8];
        corner_sums(fa, a, st);
        gather8(vels[a], nl, vel);
        fb_force_axis_plus(hg, vel, coefficient, st, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) outs[a][k * N + i] = f[k];
    }
}

// Corner forces of element i, stress plus hourglass, along axes [first, end),
// in block fixed point (block_fixed.cuh) and stored as forces_double stores
// them. Which form an axis takes depends on the geometry and on that axis'
// velocities alone, so an element's forces are the same bits however its
// axes are divided.
__device__ __forceinline__ void forces_axes(const Mesh& m, int i, int first, int end) {
    const size_t N = (size_t)m.numElem;
    int nl[8];
    load_nodelist(m.nodelist, i, nl);
    bf::ForceGeo g;
    bool ok = true;
    {
        bf::Sums s;
        double x[8];
        gather8(m.x, nl, x);
        ok &= bf::axis_sums<57, false>(x, 0, s);
        gather8(m.y, nl, x);
        ok &= bf::axis_sums<57, false>(x, 1, s);
        gather8(m.z, nl, x);
        ok &= bf::axis_sums<57, false>(x, 2, s);
        ok &= bf::force_geometry(s, g);
    }
    const double determ = LD(m.volo + i) * LD(m.v + i);
    ok &= f_gt(determ, 0.0);
    bf::ForceScale sc;
    const double coefficient = -m.prm.hgcoef * 0.01 * LD(m.ss + i) * LD(m.elemMass + i) * rcbrt_pos(determ);
    ok &= bf::force_scale(g, rcp(determ) * (1.0 / 192.0), coefficient, LD(m.p + i) + LD(m.q + i), sc);
    int again = ok ? 0 : 7;
    // one copy of the axis' code: three would not fit the instruction cache
#pragma unroll 1
    for (int a = first; a < end; ++a) {
        int64_t n[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) n[d] = a == 0 ? g.n[d][0] : a == 1 ? g.n[d][1] : g.n[d][2];
        const double* v = a == 0 ? m.xd : a == 1 ? m.yd : m.zd;
        double* out = a == 0 ? m.fsx : a == 1 ? m.fsy : m.fsz;
        double vel[8], f[8];
        gather8(v, nl, vel);
        const bool fits = bf::force_axis(g, sc, n, a == 0 ? g.unit[0] : a == 1 ? g.unit[1] : g.unit[2], vel, f);
        again |= fits ? 0 : 1 << a;
#pragma unroll
        for (int k = 0; k < 8; ++k) out[k * N + i] = f[k];
    }
    again &= (1 << end) - (1 << first);
    if (again) forces_double(m, i, again);
}
__device__ __forceinline__ void forces_elem(const Mesh& m, int i) { forces_axes(m, i, 0, 3); }
#endif

// Node n: gather in CSR order, stress then hourglass per corner
// (combineVolumeForcesTaskFunc, lulesh.cc:838-862), then the node update.
__device__ __forceinline__ void nodes_node(const Mesh& m, int n, double dt) {
    const size_t N = (size_t)m.numElem;
    const int b = LD(m.nodeElemStart + n), e = LD(m.nodeElemStart + n + 1);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for (int j = b; j < e; ++j) {
        const int c = LD(m.nodeElemCornerList + j);
        const size_t idx = (size_t)(c & 7) * N + (size_t)(c >> 3);
#if LULESH_EXACT
        fx += LD(m.fsx + idx);
        fx += LD(m.fhx + idx);
        fy += LD(m.fsy + idx);
        fy += LD(m.fhy + idx);
        fz += LD(m.fsz + idx);
        fz += LD(m.fhz + idx);
#else
        fx += LD(m.fsx + idx);  // stress + hourglass, combined by forces_elem
        fy += LD(m.fsy + idx);
        fz += LD(m.fsz + idx);
#endif
    }
    node_update(m, n, fx, fy, fz, dt);
}

// CalcKinematicsForElemsTask (lulesh.cc:1169-1275) and
// CalcMonotonicQGradientsForElemsTask (lulesh.cc:1277-1418) of element i:
// both read the same updated node positions and velocities.
#if LULESH_EXACT
__device__ __forceinline__ void kinematics_elem(const Mesh& m, int i, double dt) {
    int nl[8];
    load_nodelist(m.nodelist, i, nl);
    double x[8], y[8], z[8], xv[8], yv[8], zv[8];
    gather8(m.x, nl, x);
    gather8(m.y, nl, y);
    gather8(m.z, nl, z);
    const double volume = hex_volume(x, y, z);
    const double relv = quot_refined(volume, LD(m.volo + i));
    const double vold = m.v[i];
    m.vnew[i] = relv;
    m.delv[i] = relv - vold;
    m.arealg[i] = char_length(x, y, z, volume);

    gather8(m.xd, nl, xv);
    gather8(m.yd, nl, yv);
    gather8(m.zd, nl, zv);
    double g[6];
    m.vdov[i] = gradients_vdov(x, y, z, xv, yv, zv, LD(m.volo + i) * relv, 0.5 * dt, g);
    m.dvxi[i] = g[0];
    m.dveta[i] = g[1];
    m.dvzeta[i] = g[2];
    m.dxxi[i] = g[3];
    m.dxeta[i] = g[4];
    m.dxzeta[i] = g[5];
    update_volume(m, i, vold, relv);
}
#else
// Kinematics of element i in double: the path of the elements that do not fit
// the block fixed point of kinematics_elem. The characteristic length
// 4 V / sqrt(largest face measure) comes from the faces' t x s: the
// reference's face measure is 4 |t x s|^2 (Lagrange's identity).
// Parts: kKinGeometry stores what follows from the coordinates (and v),
// kKinVelocity what needs the velocities too.
constexpr int kKinGeometry = 1, kKinVelocity = 2;
__device__ __noinline__ void kinematics_double(const Mesh& m, int i, double dt, int parts) {
    int nl[8];
    load_nodelist(m.nodelist, i, nl);
    double x[8], y[8], z[8], xv[8], yv[8], zv[8];
    gather8(m.x, nl, x);
    gather8(m.y, nl, y);
    gather8(m.z, nl, z);
    gather8(m.xd, nl, xv);
    gather8(m.yd, nl, yv);
    gather8(m.zd, nl, zv);
    const double volume = hex_volume(x, y, z);
    const double relv = quot_refined(volume, LD(m.volo + i));
    double gr[6];
    const double vdov = gradients_vdov(x, y, z, xv, yv, zv, pmul(LD(m.volo + i), relv), 0.5 * dt, gr);
    if (parts & kKinGeometry) {
        const double vold = m.v[i];
        m.vnew[i] = relv;
        m.delv[i] = relv - vold;
        m.arealg[i] = char_length(x, y, z, volume);
        m.dxxi[i] = gr[3];
        m.dxeta[i] = gr[4];
        m.dxzeta[i] = gr[5];
        update_volume(m, i, vold, relv);
    }
    if (parts & kKinVelocity) {
        m.vdov[i] = vdov;
        m.dvxi[i] = gr[0];
        m.dveta[i] = gr[1];
        m.dvzeta[i] = gr[2];
    }
}

// Ulps (halved below 1) that the relative volume of an element at rest may
// be off 1, see kinematics_elem.
constexpr unsigned long long kUlpsBelow = 8, kUlpsAbove = 4;

// Kinematics of element i in block fixed point (block_fixed.cuh). The
// volume is closer to the exact one than the double formula that made volo,
// so an element that has not moved would come out a few ulps from 1; a
// relative volume within the rounding of that formula of 1 is 1, as in the
// reference (a delv of an ulp would send its EOS passes down the compressing
// branch).
// PARTS: the parts to form and store (kinematics_double). Which form a part
// takes depends on its own inputs alone, so an element's values are the same
// bits however its parts are divided.
template <int PARTS>
__device__ __forceinline__ void kinematics_parts(const Mesh& m, int i, double dt) {
    int nl[8];
    load_nodelist(m.nodelist, i, nl);
    bf::KinGeo g;
    bool geo = true, vel = true;
    {
        bf::Sums s;
        double x[8];
        gather8(m.x, nl, x);
        geo &= bf::axis_sums<58, false>(x, 0, s);
        gather8(m.y, nl, x);
        geo &= bf::axis_sums<58, false>(x, 1, s);
        gather8(m.z, nl, x);
        geo &= bf::axis_sums<58, false>(x, 2, s);
        geo &= bf::kin_geometry(s, g);
    }
    const double volo = LD(m.volo + i);
    const double volume = g.vol192 * (1.0 / 192.0);
    double relv = quot_refined(volume, volo);
    if (static_cast<unsigned long long>(dbits(relv) - dbits(1.0) + kUlpsBelow) <= kUlpsBelow + kUlpsAbove) relv = 1.0;
    const double vol = pmul(volo, relv);
    if ((PARTS & kKinGeometry) && geo) {
        const double vold = m.v[i], vol16 = 16.0 * vol;
        m.vnew[i] = relv;
        m.delv[i] = relv - vold;
        m.arealg[i] = pmul(16.0 * volume, rsqrt(g.face2));
        m.dxxi[i] = pmul(vol16, rsqrt(g.cc[0] + 256.0 * 1.e-36));
        m.dxeta[i] = pmul(vol16, rsqrt(g.cc[1] + 256.0 * 1.e-36));
        m.dxzeta[i] = pmul(vol16, rsqrt(g.cc[2] + 256.0 * 1.e-36));
        update_volume(m, i, vold, relv);
    }
    if (PARTS & kKinVelocity) {
        bf::VelSums v;
        double x[8];
        gather8(m.xd, nl, x);
        vel &= bf::vel_sums(x, 0, v);
        gather8(m.yd, nl, x);
        vel &= bf::vel_sums(x, 1, v);
        gather8(m.zd, nl, x);
        vel &= bf::vel_sums(x, 2, v);
        vel &= geo;
        bf::KinVel kv;
        bf::kin_velocity(g, v, kv);
        if (vel) {
            const double n64 = rcp(vol + 1.e-36) * 0.015625;
            m.dvxi[i] = pmul(kv.cv[0], n64);
            m.dveta[i] = pmul(kv.cv[1], n64);
            m.dvzeta[i] = pmul(kv.cv[2], n64);
            const double t = 0.5 * dt, b = kv.cv[0] + kv.cv[1] + kv.cv[2];
            const double num = fma(t, fma(3.0 * t, kv.detv, -2.0 * kv.ak), b);
            const double den = fma(-t, fma(-t, fma(-t, kv.detv, kv.ak), b), g.det);
            m.vdov[i] = quot(num, den);
        }
    }
    const int again = PARTS & ((geo ? 0 : kKinGeometry) | (vel ? 0 : kKinVelocity));
    if (again) kinematics_double(m, i, dt, again);
}
__device__ __forceinline__ void kinematics_elem(const Mesh& m, int i, double dt) {
    kinematics_parts<kKinGeometry | kKinVelocity>(m, i, dt);
}
#endif

// Material phase of an element by several lanes (material_share).
template <bool SPREAD, class Dt>
__device__ __forceinline__ void material_elem(const Mesh& m, int t, int r, int lanes, Dt& dt) {
    material_share<SPREAD>(m, t, r, lanes, m.dvxi, m.dveta, m.dvzeta, m.dxxi, m.dxeta, m.dxzeta, dt);
}

// --- single-problem kernels -------------------------------------------------

// Resident blocks of 128 per SM asked of the compiler. The fast variant's
// block fixed point is bound by the integer multiply and add pipes, with room
// for warps up to 128 registers: at s=150 k_forces takes 0.78, 0.82, 0.83 ms
// with 4, 5, 6 blocks, k_kinematics 0.643, 0.633, 0.641. The exact variant's
// out-of-line products leave a warp waiting on their chains: at s=60 k_forces
// takes 0.594, 0.62, 0.536, 0.661 ms with 1 to 4 blocks, k_kinematics 0.274,
// 0.274, 0.277, 0.282 (before its compares were integers; now 0.277 with 3).
constexpr int kForceBlocks = LULESH_EXACT ? 3 : 4, kKinBlocks = LULESH_EXACT ? 3 : 5;

#if !LULESH_EXACT
// The same for few elements: one axis of an element to a thread (blockIdx.y),
// and one part of its kinematics. The geometry is formed again for each, but
// a mesh that leaves the multiprocessors idle takes as long as one thread.
__global__ void __launch_bounds__(kForceBlock, kForceBlocks) k_forces_axis(Mesh m, int first, int end) {
    if (m.dtime && !m.dtime->active) return;
    const int i = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (i < end) forces_axes(m, i, blockIdx.y, blockIdx.y + 1);
}
__global__ void __launch_bounds__(kKinBlock, kKinBlocks) k_kinematics_part(Mesh m, double dt, int first, int end) {
    if (m.dtime) {
        if (!m.dtime->active) return;
        dt = m.dtime->deltatime;
    }
    const int i = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    if (blockIdx.y == 0) kinematics_parts<kKinGeometry>(m, i, dt);
    else kinematics_parts<kKinVelocity>(m, i, dt);
}
#endif

// all elements, or (RANGED) elements [first, end)
template <bool RANGED>
__global__ void __launch_bounds__(kForceBlock, kForceBlocks) k_forces(Mesh m, int first, int end) {
    if (m.dtime && !m.dtime->active) return;
    const int i = (RANGED ? first : 0) + blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (RANGED ? end : m.numElem)) forces_elem(m, i);
}

__global__ void __launch_bounds__(kNodeBlock) k_nodes(Mesh m, double dt) {
    if (m.dtime) {
        if (!m.dtime->active) return;
        dt = m.dtime->deltatime;
    }
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < m.numNode) nodes_node(m, n, dt);
}

// all elements, or (RANGED) elements [first, end)
template <bool RANGED>
__global__ void __launch_bounds__(kKinBlock, kKinBlocks) k_kinematics(Mesh m, double dt, int first, int end) {
    if (m.dtime) {
        if (!m.dtime->active) return;
        dt = m.dtime->deltatime;
    }
    const int i = (RANGED ? first : 0) + blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (RANGED ? end : m.numElem)) kinematics_elem(m, i, dt);
}

// Elements visited in repeat-count order so a warp's lanes run the same
// number of EOS passes; the dt minima end in a last-block reduction. Exact
// variant: 8 blocks of 128 per SM (64 registers), the passes being a chain of
// dependent operations (s=60: 0.266 ms, 7 and 6 blocks 0.286 and 0.295). Fast
// variant: 6 (80 registers): its integer passes are bound by the ALU pipe, and
// more blocks spill (5 to 8: s=150 0.645, 0.628, 0.627, 0.652 ms, s=45 0.0416,
// 0.0421, 0.0430, 0.0440).
constexpr int kMatBlocks = LULESH_EXACT ? 8 : 6;
// SPREAD: some class has several lanes per element (MatPlan).
template <bool SPREAD>
__global__ void __launch_bounds__(kMatBlock, kMatBlocks) k_material(Mesh m, const __grid_constant__ MatPlan plan) {
    if (m.dtime && !m.dtime->active) return;
    DtMin<LULESH_EXACT> dt;
    if (SPREAD) {
        const int nwarps = gridDim.x * (kMatBlock / 32);
        for (int w = blockIdx.x * (kMatBlock / 32) + (threadIdx.x >> 5); w < plan.warps; w += nwarps) {
            int k = 0;
            while (k + 1 < plan.n && w >= plan.cls[k + 1].warp0) ++k;
            int t, r;
            material_place(plan.cls[k], w - plan.cls[k].warp0, t, r);
            material_elem<true>(m, t, r, plan.cls[k].lanes, dt);
        }
    } else {
        const int lane = threadIdx.x & 31;
        for (int t = blockIdx.x * kMatBlock + threadIdx.x - lane; t < plan.count; t += gridDim.x * kMatBlock)
            material_elem<false>(m, plan.cls[0].first + min(t + lane, plan.count - 1), t + lane < plan.count ? 0 : 1, 1, dt);
    }
    finish_dt_reduction(m, dt.dtc, dt.dth);
}

// Up to this many elements the forces' axes, and the kinematics' parts, go to
// threads of their own: forces s=12 14.7 -> 10.5 us, s=20 14.7 -> 12.5, s=27
// (19,683) 17.7 -> 16.2, s=30 the same, s=34 20.8 -> 22.8; kinematics s=12
// 14.3 -> 11.9, s=27 16.4 -> 15.3, s=30 (27,000) 16.4 -> 16.2, s=37 18.4 ->
// 20.4.
constexpr int kSplitElems = LULESH_EXACT ? 0 : 20000, kSplitKinElems = LULESH_EXACT ? 0 : 30000;

int launch_forces_range(const Mesh& m, int first, int end, cudaStream_t s) {
    const int n = end - first, blocks = blocks_for(n, kForceBlock);
    if (n <= 0) return 0;
#if !LULESH_EXACT
    if (n <= kSplitElems) {
        k_forces_axis<<<dim3(blocks, 3), kForceBlock, 0, s>>>(m, first, end);
        return 1;
    }
#endif
    if (n == m.numElem) k_forces<false><<<blocks, kForceBlock, 0, s>>>(m, 0, n);
    else k_forces<true><<<blocks, kForceBlock, 0, s>>>(m, first, end);
    return 1;
}
int launch_forces(const Mesh& m, cudaStream_t s) { return launch_forces_range(m, 0, m.numElem, s); }
int launch_nodes(const Mesh& m, double dt, cudaStream_t s) {
    const int blocks = blocks_for(m.numNode, kNodeBlock);
    k_nodes<<<blocks, kNodeBlock, 0, s>>>(m, dt);
    return 1;
}
int launch_kinematics_range(const Mesh& m, double dt, int first, int end, cudaStream_t s) {
    const int n = end - first, blocks = blocks_for(n, kKinBlock);
    if (n <= 0) return 0;
#if !LULESH_EXACT
    if (n <= kSplitKinElems) {
        k_kinematics_part<<<dim3(blocks, 2), kKinBlock, 0, s>>>(m, dt, first, end);
        return 1;
    }
#endif
    if (n == m.numElem) k_kinematics<false><<<blocks, kKinBlock, 0, s>>>(m, dt, 0, n);
    else k_kinematics<true><<<blocks, kKinBlock, 0, s>>>(m, dt, first, end);
    return 1;
}
int launch_kinematics(const Mesh& m, double dt, cudaStream_t s) {
    return launch_kinematics_range(m, dt, 0, m.numElem, s);
}
int launch_material(const Mesh& m, const MatPlan& plan, cudaStream_t s) {
    if (plan.spread) k_material<true><<<plan.grid, kMatBlock, 0, s>>>(m, plan);
    else k_material<false><<<plan.grid, kMatBlock, 0, s>>>(m, plan);
    return 1;
}

}  // namespace LULESH_VARIANT
}  // namespace lulesh

#include "batch_kernels.cuh"
