// GPU re-voxelizer of a spinning part (crates/cfd/src/shader.rs:865-1104):
// every step the part's triangles, rotated to the step's angle, are tested
// against the lattice links around them (k_tri_scatter, nearest and farthest
// hit and hit count per link, by atomics into a per-link scratch); then every
// cell of the swept box is classified (k_voxelize): solid or fluid from the
// body-frame occupancy grid, cut links and q from the scratch, a refill of
// the populations a just-uncovered cell would have sent out, and the momentum
// the part takes from cells it covers or gives to cells it uncovers; it
// also resets the scratch of the next step.
//
// The geometric arithmetic is f32 rounded operation by operation (no fused
// multiply-add, IEEE division and square root), as the reference states it,
// so every cell asks "is this cell solid?" with the same arithmetic for
// itself and its neighbours (a disagreement would let a fluid cell read
// populations a solid cell never wrote), and the CPU oracle reproduces the
// classification bit for bit.
#pragma once

#include "lbm_device.cuh"
#include "pdl.cuh"
#include "spin_math.cuh"

namespace lbm {
namespace rv {

__device__ __forceinline__ bool occ_at(const LatParams &p, V3 b) { return occ_bit(p.occ, p.occ_lo, p.occ_invh, p.occ_n, b); }
// shader.rs:877-881
__device__ __forceinline__ bool solid_at(const LatParams &p, const StepParams &s, int x, int y, int z, bool before) {
    const V3 pc = {fs((float)x, p.kf.center[0]), fs((float)y, p.kf.center[1]), fs((float)z, p.kf.center[2])};
    return occ_at(p, to_body(before ? s.rot_prev : s.rot, pc));
}

// The link scratch: per set, 9 links x (nearest t, farthest t, hits), each a
// row of one word per box cell, so that a warp's cells read whole sectors (by
// cell, 27 words apart, every load touched 32 of them).  Two sets take turns:
// k_voxelize reads one and resets the other (shader.rs:942-948).  256x128x128
// rotor, 113 k box cells: k_voxelize 44 us and a reset kernel before, 24 us.
__device__ __forceinline__ uint32_t *link_scratch(const LatParams &p, uint32_t set) { return p.qscr + (uint64_t)set * 27u * p.nrec; }

// Whether the cells of the swept box and the layer around it are solid now
// (bit 0) and were before (bit 1): one byte per cell, written beside the
// triangle scatter, so that k_voxelize looks its neighbours up instead of
// rotating each into the body frame again (18 times a cell).
__device__ __forceinline__ uint32_t solid_index(const uint32_t *box_n, int lx, int ly, int lz) {
    return ((uint32_t)(lz + 1) * (box_n[1] + 2u) + (uint32_t)(ly + 1)) * (box_n[0] + 2u) + (uint32_t)(lx + 1);
}
__device__ __forceinline__ void solid_cell(const LatParams &p, const StepParams &s, uint32_t q) {
    const uint32_t nx = p.box_n[0] + 2u, ny = p.box_n[1] + 2u, nz = p.box_n[2] + 2u;
    if (q >= nx * ny * nz) return;
    const int x = (int)(q % nx) - 1 + p.box_lo[0], y = (int)(q / nx % ny) - 1 + p.box_lo[1], z = (int)(q / (nx * ny)) - 1 + p.box_lo[2];
    p.sol[q] = (uint8_t)((solid_at(p, s, x, y, z, false) ? 1 : 0) | (solid_at(p, s, x, y, z, true) ? 2 : 0));
}

}  // namespace rv

// shader.rs:902-940: one thread per triangle
__global__ void __launch_bounds__(BLOCK) k_tri_scatter(const __grid_constant__ LatParams p, const __grid_constant__ StepParams s) {
    using namespace rv;
    pdl_wait();
    // one warp per triangle, its lanes over the lattice points near it
    // (the blocks past the triangles' classify the box's cells)
    const uint32_t tri_blocks = (uint32_t)(((uint64_t)p.ntri * 32u + BLOCK - 1) / BLOCK);
    if (blockIdx.x >= tri_blocks) {
        solid_cell(p, s, (blockIdx.x - tri_blocks) * BLOCK + threadIdx.x);
        return;
    }
    const uint32_t t = (blockIdx.x * BLOCK + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (t >= p.ntri) return;
    const float4 t0 = p.tris[3 * t], t1 = p.tris[3 * t + 1], t2 = p.tris[3 * t + 2];
    const V3 ctr = {p.kf.center[0], p.kf.center[1], p.kf.center[2]};
    const V3 a = add(ctr, from_body(s.rot, {t0.x, t0.y, t0.z}));
    const V3 e1 = from_body(s.rot, {t1.x, t1.y, t1.z});
    const V3 e2 = from_body(s.rot, {t2.x, t2.y, t2.z});
    const V3 nrm = cross(e1, e2);
    const float nl = __fsqrt_rn(dot(nrm, nrm));
    if (nl < 1e-12f) return;
    const V3 nn = {__fdiv_rn(nrm.x, nl), __fdiv_rn(nrm.y, nl), __fdiv_rn(nrm.z, nl)};
    const V3 b = add(a, e1), c = add(a, e2);
    const int lo[3] = {max((int)ceilf(fs(fminf(fminf(a.x, b.x), c.x), 1.415f)), p.box_lo[0]),
                       max((int)ceilf(fs(fminf(fminf(a.y, b.y), c.y), 1.415f)), p.box_lo[1]),
                       max((int)ceilf(fs(fminf(fminf(a.z, b.z), c.z), 1.415f)), p.box_lo[2])};
    const int hi[3] = {min((int)floorf(fa(fmaxf(fmaxf(a.x, b.x), c.x), 1.415f)), p.box_lo[0] + (int)p.box_n[0] - 1),
                       min((int)floorf(fa(fmaxf(fmaxf(a.y, b.y), c.y), 1.415f)), p.box_lo[1] + (int)p.box_n[1] - 1),
                       min((int)floorf(fa(fmaxf(fmaxf(a.z, b.z), c.z), 1.415f)), p.box_lo[2] + (int)p.box_n[2] - 1)};
    const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1;
    const int npts = (nx > 0 && ny > 0 && nz > 0) ? nx * ny * nz : 0;
    uint32_t *scr = link_scratch(p, s.scr);
    for (int q = (int)lane; q < npts; q += 32) {
                const int x = lo[0] + q % nx, y = lo[1] + (q / nx) % ny, z = lo[2] + q / (nx * ny);
                const V3 pt = {(float)x, (float)y, (float)z};
                const float d0 = dot(nn, sub(pt, a));
                if (fabsf(d0) > 1.415f) continue;
                const uint32_t k = ((uint32_t)(z - p.box_lo[2]) * p.box_n[1] + (uint32_t)(y - p.box_lo[1])) * p.box_n[0] + (uint32_t)(x - p.box_lo[0]);
#pragma unroll
                for (int i = 1; i < 19; i += 2) {
                    const V3 cv = {(float)CX(i), (float)CY(i), (float)CZ(i)};
                    const float d1 = fa(d0, dot(nn, cv));
                    if (fm(d0, d1) > 0.0f && fabsf(d0) > 1e-6f) continue;
                    const float tt = ray_tri(pt, cv, a, e1, e2);
                    if (tt <= 1.0f) {
                        uint32_t *q0 = scr + (uint64_t)(3 * ((i - 1) / 2)) * p.nrec + k;
                        const uint32_t tb = __float_as_uint(tt > 0.0f ? tt : 0.0f);
                        atomicMin(q0, tb);
                        atomicMax(q0 + p.nrec, tb);
                        atomicAdd(q0 + 2ull * p.nrec, 1u);
                    }
                }
            }
}

// shader.rs:953-1104: one thread per swept-box cell (record k); Q is the
// parity of the previous step (the refill writes what the cell would have
// sent out then)
template <class S, int Q>
__global__ void __launch_bounds__(BLOCK) k_voxelize(const __grid_constant__ LatParams p, const __grid_constant__ StepParams s) {
    using namespace rv;
    using R = typename Pop<S>::real;
    pdl_wait();
    const uint32_t k0 = blockIdx.x * BLOCK + threadIdx.x;
    const bool live = k0 < p.nrec;
    const uint32_t k = live ? k0 : p.nrec - 1;  // (idle threads only help their warp)
    // the other set, read by the step before, is reset for the next one
    uint32_t *scr = link_scratch(p, s.scr), *next = link_scratch(p, s.scr ^ 1u);
#pragma unroll
    for (int w = 0; w < 27; w++)
        if (live) next[(uint64_t)w * p.nrec + k] = w % 3 == 0 ? 0x7f7fffffu : 0u;
    const uint32_t lx = k % p.box_n[0], ly = (k / p.box_n[0]) % p.box_n[1], lz = k / (p.box_n[0] * p.box_n[1]);
    const int px = (int)lx + p.box_lo[0], py = (int)ly + p.box_lo[1], pz = (int)lz + p.box_lo[2];
    const uint32_t n = ((uint32_t)pz * p.NY + (uint32_t)py) * p.NX + (uint32_t)px;
    const Consts<R> &kk = K<R>(p);
    const R pc[3] = {(R)px - kk.center[0], (R)py - kk.center[1], (R)pz - kk.center[2]};
    const uint32_t sq = solid_index(p.box_n, (int)lx, (int)ly, (int)lz);
    const bool solid_now = (p.sol[sq] & 1u) != 0, solid_before = (p.sol[sq] & 2u) != 0;
    // Refill of the cells uncovered this step: the density and the mean
    // non-equilibrium stress of the neighbours that are fluid now and were
    // before.  Few cells need it, but one thread walking its 18 neighbours (two
    // occupancy tests and a record each, one after another) took most of the
    // kernel's time: the warp takes one such cell at a time, a lane per
    // neighbour, and the lanes' terms are added in the neighbours' order.
    // 256x128x128 rotor: 45 -> 16 us.
    R rs = 0, cnt = 0, pis[6] = {0, 0, 0, 0, 0, 0};
    const bool refill = live && !solid_now && solid_before;
    for (uint32_t todo = __ballot_sync(0xffffffffu, refill); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1, lane = (int)(threadIdx.x & 31u), i = lane + 1;
        const int ax = __shfl_sync(0xffffffffu, px, src), ay = __shfl_sync(0xffffffffu, py, src), az = __shfl_sync(0xffffffffu, pz, src);
        bool ok = false;
        R t[7] = {0, 0, 0, 0, 0, 0, 0};
        if (lane < 18) {
            const int nx = ax + CX(i), ny = ay + CY(i), nz = az + CZ(i);
            const int qxl = nx - p.box_lo[0], qyl = ny - p.box_lo[1], qzl = nz - p.box_lo[2];
            ok = p.sol[solid_index(p.box_n, qxl, qyl, qzl)] == 0 && qxl >= 0 && qyl >= 0 && qzl >= 0 && qxl < (int)p.box_n[0] && qyl < (int)p.box_n[1] &&
                 qzl < (int)p.box_n[2];
            if (ok) {
                const uint32_t k2 = ((uint32_t)qzl * p.box_n[1] + (uint32_t)qyl) * p.box_n[0] + (uint32_t)qxl;
                R fp[19];
                fp[0] = 0;
                for (int j = 1; j < 19; j++) fp[j] = Rec<R>::fpost(p, k2, j);
                const Moments<R> m2 = moments<R>(fp);
                const R r2 = Rec<R>::macro(p, k2, 0);
                const R u2[3] = {Rec<R>::macro(p, k2, 1), Rec<R>::macro(p, k2, 2), Rec<R>::macro(p, k2, 3)};
                const R tr = (m2.sxx + m2.syy + m2.szz) / (R)3;
                const R uu = u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2];
                t[0] = m2.sxx - tr - r2 * (u2[0] * u2[0] - uu / (R)3);
                t[1] = m2.syy - tr - r2 * (u2[1] * u2[1] - uu / (R)3);
                t[2] = m2.szz - tr - r2 * (u2[2] * u2[2] - uu / (R)3);
                t[3] = m2.sxy - r2 * u2[0] * u2[1];
                t[4] = m2.sxz - r2 * u2[0] * u2[2];
                t[5] = m2.syz - r2 * u2[1] * u2[2];
                t[6] = r2;
            }
        }
        const uint32_t use = __ballot_sync(0xffffffffu, ok);
        for (int q = 0; q < 18; q++) {
            if (!(use >> q & 1u)) continue;
            R v[7];
#pragma unroll
            for (int j = 0; j < 7; j++) v[j] = __shfl_sync(0xffffffffu, t[j], q);
            if (lane == src) {
                rs += v[6];
                cnt += (R)1;
#pragma unroll
                for (int j = 0; j < 6; j++) pis[j] += v[j];
            }
        }
    }
    if (!live) return;
    R F[3] = {0, 0, 0};
    if (solid_now) {
        p.flags[n] = 1u | ((k + 1u) << 2);
        p.recs[k * RS + R_MASK] = 0u;
        if (!solid_before) {
            // covered this step: the part takes the cell's momentum
            const R rho = Rec<R>::macro(p, k, 0);
            for (int a = 0; a < 3; a++) F[a] = rho * Rec<R>::macro(p, k, 1 + a);
        }
        const R T[3] = {pc[1] * F[2] - pc[2] * F[1], pc[2] * F[0] - pc[0] * F[2], pc[0] * F[1] - pc[1] * F[0]};
        for (int a = 0; a < 3; a++) { Rec<R>::set_ft(p, k, a, F[a]); Rec<R>::set_ft(p, k, 3 + a, T[a]); }
        return;
    }
    // link hits of this step: each link is kept once, at the cell it leaves
    // in the positive direction; the cell at its other end reads it mirrored
    float qv[19], qx[19];
    uint32_t nh[19];
#pragma unroll
    for (int i = 1; i < 19; i++) {
        qv[i] = 9.0f; qx[i] = -1.0f; nh[i] = 0u;
        if (i & 1) {
            const uint32_t *q0 = scr + (uint64_t)(3 * ((i - 1) / 2)) * p.nrec + k;
            const uint32_t c = q0[2ull * p.nrec], v0 = q0[0], v1 = q0[p.nrec];
            if (c) { qv[i] = __uint_as_float(v0); qx[i] = __uint_as_float(v1); nh[i] = c; }
        } else {
            const int qxl = (int)lx + CX(i), qyl = (int)ly + CY(i), qzl = (int)lz + CZ(i);
            if (qxl >= 0 && qyl >= 0 && qzl >= 0 && qxl < (int)p.box_n[0] && qyl < (int)p.box_n[1] && qzl < (int)p.box_n[2]) {
                const uint32_t k2 = ((uint32_t)qzl * p.box_n[1] + (uint32_t)qyl) * p.box_n[0] + (uint32_t)qxl;
                const uint32_t *q0 = scr + (uint64_t)(3 * ((i - 2) / 2)) * p.nrec + k2;
                const uint32_t c = q0[2ull * p.nrec], v0 = q0[0], v1 = q0[p.nrec];
                if (c) { qv[i] = fs(1.0f, __uint_as_float(v1)); qx[i] = fs(1.0f, __uint_as_float(v0)); nh[i] = c; }
            }
        }
    }
    uint32_t mask = 0, near = 0;  // near: the solid neighbours
    {
        const int sx = (int)p.box_n[0] + 2, sxy = sx * ((int)p.box_n[1] + 2);
#pragma unroll
        for (int i = 1; i < 19; i++) near |= (p.sol[(int)sq + CX(i) + CY(i) * sx + CZ(i) * sxy] & 1u) << i;
    }
#pragma unroll
    for (int i = 1; i < 19; i++) {
        // a wall where the neighbour is solid, or where the link crosses a
        // sheet thinner than a cell (two hits); q from the nearest hit
        if (near & (1u << i)) {
            if (nh[i] == 0u) qv[i] = 1.0f;
            mask |= 1u << i;
        } else if (nh[i] >= 2u && fs(qx[i], qv[i]) > 1e-5f) {
            mask |= 1u << i;
        } else {
            qv[i] = 1.0f;
        }
    }
    // the record's first words in 16-byte pieces (mask, cell, distances; word 11
    // starts the populations)
    static_assert(RS * 4 % 16 == 0 && R_MASK == 0 && R_CELL == 1 && R_Q == 2 && R_FPOST == 11 && R_FT == 33, "record in 16-byte pieces");
    uint32_t qw[11];
    qw[0] = mask;
    qw[1] = n;
#pragma unroll
    for (int w = 0; w < 9; w++) {
        const uint32_t lo = __half_as_ushort(__float2half_rn(fminf(qv[2 * w + 1], 1.0f)));
        const uint32_t hi = __half_as_ushort(__float2half_rn(fminf(qv[2 * w + 2], 1.0f)));
        qw[R_Q + w] = lo | (hi << 16);
    }
    {
        uint32_t *rec = p.recs + (uint64_t)k * RS;
        reinterpret_cast<uint4 *>(rec)[0] = make_uint4(qw[0], qw[1], qw[2], qw[3]);
        reinterpret_cast<uint4 *>(rec)[1] = make_uint4(qw[4], qw[5], qw[6], qw[7]);
        reinterpret_cast<uint2 *>(rec)[4] = make_uint2(qw[8], qw[9]);
        rec[10] = qw[10];
    }
    if (solid_before) {
        // uncovered this step: refill what the cell would have sent out last
        // step, the equilibrium at the wall velocity and the density of the
        // fluid neighbours plus their mean non-equilibrium stress (gathered
        // above); the part gives up the refill's momentum
        const R rho = cnt > (R)0 ? rs / cnt : (R)1;
        R om[3];
        if (sizeof(R) == 8) { om[0] = (R)s.omega_d[0]; om[1] = (R)s.omega_d[1]; om[2] = (R)s.omega_d[2]; }
        else { om[0] = (R)s.omega[0]; om[1] = (R)s.omega[1]; om[2] = (R)s.omega[2]; }
        const R uw[3] = {om[1] * pc[2] - om[2] * pc[1], om[2] * pc[0] - om[0] * pc[2], om[0] * pc[1] - om[1] * pc[0]};
        const R usq = (R)1.5 * (uw[0] * uw[0] + uw[1] * uw[1] + uw[2] * uw[2]);
        R fe[19];
#pragma unroll
        for (int i = 0; i < 19; i++) fe[i] = feq_i<R>(i, rho - (R)1, rho, uw[0], uw[1], uw[2], usq);
        if (cnt > (R)0) {
            for (int j = 0; j < 6; j++) pis[j] /= cnt;
            const R tr = (pis[0] + pis[1] + pis[2]) * (R)(1.0 / 3.0);
#pragma unroll
            for (int i = 0; i < 19; i++) fe[i] += fneq_i<R>(i, pis, tr);
        }
        const Nb nb = make_nb(p, (uint32_t)px, (uint32_t)py, (uint32_t)pz);
        Rng rng{sr_hash_mix(n, s.seed_mix)};
        store_prev_out<S, Q>(p, n, nb, 0x7ffffu, fe, rng);
        for (int a = 0; a < 3; a++) F[a] = -rho * uw[a];
        for (int i = 1; i < 19; i++) Rec<R>::set_fpost(p, k, i, fe[i]);
        Rec<R>::set_macro(p, k, 0, rho);
        for (int a = 0; a < 3; a++) Rec<R>::set_macro(p, k, 1 + a, uw[a]);
    }
    const R T[3] = {pc[1] * F[2] - pc[2] * F[1], pc[2] * F[0] - pc[0] * F[2], pc[0] * F[1] - pc[1] * F[0]};
    for (int a = 0; a < 3; a++) { Rec<R>::set_ft(p, k, a, F[a]); Rec<R>::set_ft(p, k, 3 + a, T[a]); }
    p.flags[n] = (k + 1u) << 2;
}

}  // namespace lbm
