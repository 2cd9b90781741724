// Box–box SAT, pair dispatch and the XPBD contact solve (device code).
#pragma once

#include "physics.cuh"

namespace dyph {

// Branch word of a box-box contact (filled when box_box_centroid gets `br`):
//   bits 0-1  SAT axis type (0 face of A, 1 face of B, 2 edge pair)
//   bits 2-3  axis i, bits 4-5 axis j (edge pair)
//   bit  7    reference face on B (face case; after the larger-face switch)
//   bits 8-9  reference face axis
//   bits 10-17 incident vertices kept (face case)
//   bits 18-21 edge-point signs s0A, s1A, s0B, s1B negative (edge case)
//   bit  22   edge case with |1 - b12^2| > 1e-6 (closest-point parameters solved)
constexpr uint32_t kBrRefB = 1u << 7;
constexpr uint32_t kBrDenom = 1u << 22;

// box_box (core/src/narrowphase.cpp:130-306) followed by the centroid
// reduction of process_pair (:991-998). Returns false for no contact.
__device__ __forceinline__ bool box_box_centroid(float acx, float acy, float acz, const float Ae[3][3],
                                                 const float Ah[3], float bcx, float bcy, float bcz,
                                                 const float Be[3][3], const float Bh[3], Contact& out,
                                                 uint32_t* br = nullptr) {
    const float eps_par = 1e-5f;
    const float dx = bcx - acx, dy = bcy - acy, dz = bcz - acz;
    SatBest best{1e30f, -1, 0, 0, 0.f, 1.f, 0.f};
    // The axes of a group are tested together and a separating one ends the
    // pair after it, so a group's square roots and sums overlap in time: the
    // result is the same as that of a return at the first separating axis.
    {
        float ov[6], dl[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            ov[i] = sat_overlap(Ae[i][0], Ae[i][1], Ae[i][2], Ae, Ah, Be, Bh, dx, dy, dz, dl[i]);
            ov[3 + i] = sat_overlap(Be[i][0], Be[i][1], Be[i][2], Ae, Ah, Be, Bh, dx, dy, dz, dl[3 + i]);
        }
        if (ov[0] <= 0.f || ov[1] <= 0.f || ov[2] <= 0.f || ov[3] <= 0.f || ov[4] <= 0.f || ov[5] <= 0.f)
            return false;
#pragma unroll
        for (int i = 0; i < 3; ++i) sat_keep(ov[i], dl[i], Ae[i][0], Ae[i][1], Ae[i][2], 0, i, 0, best);
#pragma unroll
        for (int i = 0; i < 3; ++i) sat_keep(ov[3 + i], dl[3 + i], Be[i][0], Be[i][1], Be[i][2], 1, i, 0, best);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float ov[3], dl[3], l[3][3];
        bool apart = false;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float cx = Ae[i][1] * Be[j][2] - Ae[i][2] * Be[j][1];
            const float cy = Ae[i][2] * Be[j][0] - Ae[i][0] * Be[j][2];
            const float cz = Ae[i][0] * Be[j][1] - Ae[i][1] * Be[j][0];
            const float len2 = cx * cx + cy * cy + cz * cz;
            const bool parallel = len2 < eps_par * eps_par;  // no axis
            const float inv_l = rsqrt_ieee(parallel ? 1.f : len2);
            l[j][0] = cx * inv_l;
            l[j][1] = cy * inv_l;
            l[j][2] = cz * inv_l;
            const float o = sat_overlap(l[j][0], l[j][1], l[j][2], Ae, Ah, Be, Bh, dx, dy, dz, dl[j]);
            apart = apart || (!parallel && o <= 0.f);
            ov[j] = parallel ? 1e30f : o;
        }
        if (apart) return false;
#pragma unroll
        for (int j = 0; j < 3; ++j) sat_keep(ov[j], dl[j], l[j][0], l[j][1], l[j][2], 2, i, j, best);
    }
    const float bnx = best.nx, bny = best.ny, bnz = best.nz;
    float sx_acc = 0.f, sy_acc = 0.f, sz_acc = 0.f, sd_acc = 0.f;
    int n_out = 0;
    int best_type = best.type, best_i = best.i;
    uint32_t word = static_cast<uint32_t>(best.type) | (static_cast<uint32_t>(best.i) << 2) |
                    (static_cast<uint32_t>(best.j) << 4);
    if (best_type == 0 || best_type == 1) {
        if (best_type == 0) {
            // the B face most parallel to A's axis, if it is larger
            const float ax = pick3(best_i, Ae[0][0], Ae[1][0], Ae[2][0]);
            const float ay = pick3(best_i, Ae[0][1], Ae[1][1], Ae[2][1]);
            const float az = pick3(best_i, Ae[0][2], Ae[1][2], Ae[2][2]);
            const float c0 = fabsf(ax * Be[0][0] + ay * Be[0][1] + az * Be[0][2]);
            const float c1 = fabsf(ax * Be[1][0] + ay * Be[1][1] + az * Be[1][2]);
            const float c2 = fabsf(ax * Be[2][0] + ay * Be[2][1] + az * Be[2][2]);
            int j_best = 0;
            if (c1 > c0) j_best = 1;
            if (c2 > (j_best == 1 ? c1 : c0)) j_best = 2;
            // products of the two other half extents, in (axis + 1, axis + 2) order
            const float area_b = pick3(j_best, Bh[1] * Bh[2], Bh[2] * Bh[0], Bh[0] * Bh[1]);
            const float area_a = pick3(best_i, Ah[1] * Ah[2], Ah[2] * Ah[0], Ah[0] * Ah[1]);
            if (area_b > area_a) { best_type = 1; best_i = j_best; }
        }
        const bool a_is_ref = (best_type == 0);
        const int ref_ax = best_i;
        word |= (a_is_ref ? 0u : kBrRefB) | (static_cast<uint32_t>(ref_ax) << 8);
        const float rcx = a_is_ref ? acx : bcx, rcy = a_is_ref ? acy : bcy, rcz = a_is_ref ? acz : bcz;
        float Re[3][3], Ie[3][3], Rh[3], Ih[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                Re[r][q] = a_is_ref ? Ae[r][q] : Be[r][q];
                Ie[r][q] = a_is_ref ? Be[r][q] : Ae[r][q];
            }
            Rh[r] = a_is_ref ? Ah[r] : Bh[r];
            Ih[r] = a_is_ref ? Bh[r] : Ah[r];
        }
        const float icx = a_is_ref ? bcx : acx, icy = a_is_ref ? bcy : acy, icz = a_is_ref ? bcz : acz;
        const float rc_dot_n3 = rcx * bnx + rcy * bny + rcz * bnz;
        const float sign_depth = a_is_ref ? 1.f : -1.f;
        const float Rh_ref = pick3(ref_ax, Rh[0], Rh[1], Rh[2]);
        const float Rh_t0 = pick3(ref_ax, Rh[1], Rh[2], Rh[0]), Rh_t1 = pick3(ref_ax, Rh[2], Rh[0], Rh[1]);
        float Rt0[3], Rt1[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            Rt0[q] = pick3(ref_ax, Re[1][q], Re[2][q], Re[0][q]);
            Rt1[q] = pick3(ref_ax, Re[2][q], Re[0][q], Re[1][q]);
        }
        // half edges of the incident box: a vertex is its centre plus or minus
        // each (the reference's sign factors are exact, so a subtraction is the
        // same float)
        float E[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 3; ++q) E[r][q] = Ih[r] * Ie[r][q];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float vx = (k & 1) ? icx + E[0][0] : icx - E[0][0];
            float vy = (k & 1) ? icy + E[0][1] : icy - E[0][1];
            float vz = (k & 1) ? icz + E[0][2] : icz - E[0][2];
            vx = (k & 2) ? vx + E[1][0] : vx - E[1][0];
            vy = (k & 2) ? vy + E[1][1] : vy - E[1][1];
            vz = (k & 2) ? vz + E[1][2] : vz - E[1][2];
            vx = (k & 4) ? vx + E[2][0] : vx - E[2][0];
            vy = (k & 4) ? vy + E[2][1] : vy - E[2][1];
            vz = (k & 4) ? vz + E[2][2] : vz - E[2][2];
            const float v_dot_n = vx * bnx + vy * bny + vz * bnz;
            const float dv = Rh_ref + sign_depth * (v_dot_n - rc_dot_n3);
            const float vx_rel = vx - rcx, vy_rel = vy - rcy, vz_rel = vz - rcz;
            const float qt0 = vx_rel * Rt0[0] + vy_rel * Rt0[1] + vz_rel * Rt0[2];
            const float qt1 = vx_rel * Rt1[0] + vy_rel * Rt1[1] + vz_rel * Rt1[2];
            const bool keep = !(dv <= 0.f) && !(fabsf(qt0) > Rh_t0 + 1e-3f) && !(fabsf(qt1) > Rh_t1 + 1e-3f) && n_out < 4;
            // centroid accumulation in the reference's order (cx += opx[k] ...)
            const float cx = sx_acc + (vx - sign_depth * dv * bnx);
            const float cy = sy_acc + (vy - sign_depth * dv * bny);
            const float cz = sz_acc + (vz - sign_depth * dv * bnz);
            const float cd = sd_acc + dv;
            sx_acc = keep ? cx : sx_acc;
            sy_acc = keep ? cy : sy_acc;
            sz_acc = keep ? cz : sz_acc;
            sd_acc = keep ? cd : sd_acc;
            word |= keep ? 1u << (10 + k) : 0u;
            n_out += keep ? 1 : 0;
        }
    } else {
        const int i = best.i, j = best.j;
        // the edges' directions and the two other axes of each box, in (axis + 1, axis + 2) order
        float uA[3], uB[3], a0[3], a1[3], b0[3], b1[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            uA[q] = pick3(i, Ae[0][q], Ae[1][q], Ae[2][q]);
            a0[q] = pick3(i, Ae[1][q], Ae[2][q], Ae[0][q]);
            a1[q] = pick3(i, Ae[2][q], Ae[0][q], Ae[1][q]);
            uB[q] = pick3(j, Be[0][q], Be[1][q], Be[2][q]);
            b0[q] = pick3(j, Be[1][q], Be[2][q], Be[0][q]);
            b1[q] = pick3(j, Be[2][q], Be[0][q], Be[1][q]);
        }
        const float Ah0 = pick3(i, Ah[1], Ah[2], Ah[0]), Ah1 = pick3(i, Ah[2], Ah[0], Ah[1]);
        const float Bh0 = pick3(j, Bh[1], Bh[2], Bh[0]), Bh1 = pick3(j, Bh[2], Bh[0], Bh[1]);
        const float s0A = (-bnx * a0[0] - bny * a0[1] - bnz * a0[2]) >= 0.f ? 1.f : -1.f;
        const float s1A = (-bnx * a1[0] - bny * a1[1] - bnz * a1[2]) >= 0.f ? 1.f : -1.f;
        float pAx = acx + s0A * Ah0 * a0[0] + s1A * Ah1 * a1[0];
        float pAy = acy + s0A * Ah0 * a0[1] + s1A * Ah1 * a1[1];
        float pAz = acz + s0A * Ah0 * a0[2] + s1A * Ah1 * a1[2];
        const float s0B = (bnx * b0[0] + bny * b0[1] + bnz * b0[2]) >= 0.f ? 1.f : -1.f;
        const float s1B = (bnx * b1[0] + bny * b1[1] + bnz * b1[2]) >= 0.f ? 1.f : -1.f;
        float pBx = bcx + s0B * Bh0 * b0[0] + s1B * Bh1 * b1[0];
        float pBy = bcy + s0B * Bh0 * b0[1] + s1B * Bh1 * b1[1];
        float pBz = bcz + s0B * Bh0 * b0[2] + s1B * Bh1 * b1[2];
        const float uAx = uA[0], uAy = uA[1], uAz = uA[2];
        const float uBx = uB[0], uBy = uB[1], uBz = uB[2];
        float b12 = uAx * uBx + uAy * uBy + uAz * uBz;
        float denom = 1.f - b12 * b12;
        float wx = pAx - pBx, wy = pAy - pBy, wz = pAz - pBz;
        float d1 = wx * uAx + wy * uAy + wz * uAz;
        float d2 = wx * uBx + wy * uBy + wz * uBz;
        float s_t = 0.f, t_t = 0.f;
        word |= (s0A < 0.f ? 1u << 18 : 0u) | (s1A < 0.f ? 1u << 19 : 0u) | (s0B < 0.f ? 1u << 20 : 0u) |
                (s1B < 0.f ? 1u << 21 : 0u) | (fabsf(denom) > 1e-6f ? kBrDenom : 0u);
        if (fabsf(denom) > 1e-6f) {
            s_t = __fdiv_rn(b12 * d2 - d1, denom);
            t_t = __fdiv_rn(d2 - b12 * d1, denom);
        }
        float qAx = pAx + s_t * uAx, qAy = pAy + s_t * uAy, qAz = pAz + s_t * uAz;
        float qBx = pBx + t_t * uBx, qBy = pBy + t_t * uBy, qBz = pBz + t_t * uBz;
        sx_acc = 0.f + 0.5f * (qAx + qBx);
        sy_acc = 0.f + 0.5f * (qAy + qBy);
        sz_acc = 0.f + 0.5f * (qAz + qBz);
        sd_acc = 0.f + best.ov;
        n_out = 1;
    }
    if (n_out == 0) return false;
    if (br) *br = word;
    float inv = __frcp_rn(static_cast<float>(n_out));
    out.px = sx_acc * inv; out.py = sy_acc * inv; out.pz = sz_acc * inv;
    out.nx = bnx; out.ny = bny; out.nz = bnz;
    out.depth = sd_acc * inv;
    return true;
}

// process_pair for box / sphere shapes (narrowphase.cpp:920-1001).
// Returns true and fills `c` when the pair is in contact.
template <class Bodies, class Shapes>
__device__ __forceinline__ bool process_pair(const Bodies& B, const Shapes& S, uint32_t ia, uint32_t ib, Contact& c,
                                             uint32_t* br = nullptr) {
    const uint32_t sha = B.shape(ia), shb = B.shape(ib);
    const uint32_t ta = S.type(sha), tb = S.type(shb);
    c.a = ia; c.b = ib;
    if (ta == kShapeSphere && tb == kShapeSphere)
        return sphere_sphere(B.px(ia), B.py(ia), B.pz(ia), S.hx(sha), B.px(ib), B.py(ib), B.pz(ib), S.hx(shb), c, br);
    if ((ta == kShapeSphere && tb == kShapeBox) || (ta == kShapeBox && tb == kShapeSphere)) {
        // one path for both orders, the normal flipped when the sphere comes first
        const bool first = ta == kShapeSphere;
        const uint32_t is = first ? ia : ib, ibx = first ? ib : ia, shs = first ? sha : shb, shx = first ? shb : sha;
        float E[3][3];
        make_axes(B.qw(ibx), B.qx(ibx), B.qy(ibx), B.qz(ibx), E);
        if (!sphere_box(B.px(is), B.py(is), B.pz(is), S.hx(shs), B.px(ibx), B.py(ibx), B.pz(ibx), E, S.hx(shx),
                        S.hy(shx), S.hz(shx), c, br))
            return false;
        if (first) { c.nx = -c.nx; c.ny = -c.ny; c.nz = -c.nz; }
        return true;
    }
    if (ta == kShapeBox && tb == kShapeBox) {
        float Ae[3][3], Be[3][3];
        const float Ah[3] = {S.hx(sha), S.hy(sha), S.hz(sha)};
        const float Bh[3] = {S.hx(shb), S.hy(shb), S.hz(shb)};
        make_axes(B.qw(ia), B.qx(ia), B.qy(ia), B.qz(ia), Ae);
        make_axes(B.qw(ib), B.qx(ib), B.qy(ib), B.qz(ib), Be);
        return box_box_centroid(B.px(ia), B.py(ia), B.pz(ia), Ae, Ah, B.px(ib), B.py(ib), B.pz(ib), Be, Bh, c, br);
    }
    return false;  // convex hulls / meshes are not on this path
}

// ── XPBD contact solve (core/src/xpbd_solver.cpp:40-133, 413-521) ──────────

template <class Bodies>
__device__ __forceinline__ void world_inv_inertia(const Bodies& B, uint32_t bi, float vx, float vy, float vz,
                                                  float& ox, float& oy, float& oz) {
    const float qw = B.qw(bi), qx = B.qx(bi), qy = B.qy(bi), qz = B.qz(bi);
    const float R00 = 1.f - 2.f * (qy * qy + qz * qz), R01 = 2.f * (qx * qy + qz * qw), R02 = 2.f * (qx * qz - qy * qw);
    const float R10 = 2.f * (qx * qy - qz * qw), R11 = 1.f - 2.f * (qx * qx + qz * qz), R12 = 2.f * (qy * qz + qx * qw);
    const float R20 = 2.f * (qx * qz + qy * qw), R21 = 2.f * (qy * qz - qx * qw), R22 = 1.f - 2.f * (qx * qx + qy * qy);
    const float lx = R00 * vx + R10 * vy + R20 * vz;
    const float ly = R01 * vx + R11 * vy + R21 * vz;
    const float lz = R02 * vx + R12 * vy + R22 * vz;
    const float ixx = B.ixx(bi), iyy = B.iyy(bi), izz = B.izz(bi);
    const float ixy = B.ixy(bi), ixz = B.ixz(bi), iyz = B.iyz(bi);
    const float ilx = ixx * lx + ixy * ly + ixz * lz;
    const float ily = ixy * lx + iyy * ly + iyz * lz;
    const float ilz = ixz * lx + iyz * ly + izz * lz;
    ox = R00 * ilx + R01 * ily + R02 * ilz;
    oy = R10 * ilx + R11 * ily + R12 * ilz;
    oz = R20 * ilx + R21 * ily + R22 * ilz;
}

template <class Bodies>
__device__ __forceinline__ void apply_ang_delta(const Bodies& B, uint32_t bi, float ax, float ay, float az) {
    if (B.im(bi) == 0.f) return;
    const float qw = B.qw(bi), qx = B.qx(bi), qy = B.qy(bi), qz = B.qz(bi);
    B.qw(bi) += 0.5f * (-ax * qx - ay * qy - az * qz);
    B.qx(bi) += 0.5f * (ax * qw + ay * qz - az * qy);
    B.qy(bi) += 0.5f * (-ax * qz + ay * qw + az * qx);
    B.qz(bi) += 0.5f * (ax * qy - ay * qx + az * qw);
}

// Result codes of one contact solve.
constexpr int kSolveSkipped = 0;   // depth <= 0 or already resolved
constexpr int kSolveDone = 1;      // correction applied
constexpr int kSolveDeferred = 2;  // w_total < 1e-10: lambda untouched, retried next iteration

// Branch flags of one contact solve (solve_contact's optional `flags`).
constexpr uint32_t kSfActive = 1u;     // position correction applied
constexpr uint32_t kSfNormal = 2u;     // normal velocity impulse (vrel_n < 0)
constexpr uint32_t kSfFriction = 4u;   // friction impulse applied
constexpr uint32_t kSfClamped = 8u;    // friction impulse clamped to mu * j_n_static

template <class Bodies>
__device__ __forceinline__ int solve_contact(const Bodies& B, const Contact& ct, float mu, float& lc, float dt,
                                             uint32_t* flags = nullptr) {
    const uint32_t ia = ct.a, ib = ct.b;
    const float depth = ct.depth;
    if (depth <= 0.f) return kSolveSkipped;
    const float remaining = depth - lc;
    if (remaining <= 1e-6f) return kSolveSkipped;
    const float nx = ct.nx, ny = ct.ny, nz = ct.nz;
    const float px = ct.px, py = ct.py, pz = ct.pz;
    const float wa = B.im(ia), wb = B.im(ib);
    const float rax = px - B.px(ia), ray = py - B.py(ia), raz = pz - B.pz(ia);
    const float rbx = px - B.px(ib), rby = py - B.py(ib), rbz = pz - B.pz(ib);
    const float raxnx = ray * nz - raz * ny, raxny = raz * nx - rax * nz, raxnz = rax * ny - ray * nx;
    const float rbxnx = rby * nz - rbz * ny, rbxny = rbz * nx - rbx * nz, rbxnz = rbx * ny - rby * nx;
    float iIa_x, iIa_y, iIa_z, iIb_x, iIb_y, iIb_z;
    world_inv_inertia(B, ia, raxnx, raxny, raxnz, iIa_x, iIa_y, iIa_z);
    world_inv_inertia(B, ib, rbxnx, rbxny, rbxnz, iIb_x, iIb_y, iIb_z);
    const float wa_ang = raxnx * iIa_x + raxny * iIa_y + raxnz * iIa_z;
    const float wb_ang = rbxnx * iIb_x + rbxny * iIb_y + rbxnz * iIb_z;
    const float w_total = wa + wb + wa_ang + wb_ang;
    if (w_total < 1e-10f) return kSolveDeferred;
    const float dl = __fdiv_rn(remaining, w_total);
    lc += remaining;
    if (flags) *flags = kSfActive;
    if (wa != 0.f) { B.px(ia) += wa * dl * nx; B.py(ia) += wa * dl * ny; B.pz(ia) += wa * dl * nz; }
    if (wb != 0.f) { B.px(ib) -= wb * dl * nx; B.py(ib) -= wb * dl * ny; B.pz(ib) -= wb * dl * nz; }
    apply_ang_delta(B, ia, dl * iIa_x, dl * iIa_y, dl * iIa_z);
    apply_ang_delta(B, ib, -dl * iIb_x, -dl * iIb_y, -dl * iIb_z);
    {
        const float oax = B.wx(ia), oay = B.wy(ia), oaz = B.wz(ia);
        const float obx = B.wx(ib), oby = B.wy(ib), obz = B.wz(ib);
        const float vcax = B.vx(ia) + oay * raz - oaz * ray;
        const float vcay = B.vy(ia) + oaz * rax - oax * raz;
        const float vcaz = B.vz(ia) + oax * ray - oay * rax;
        const float vcbx = B.vx(ib) + oby * rbz - obz * rby;
        const float vcby = B.vy(ib) + obz * rbx - obx * rbz;
        const float vcbz = B.vz(ib) + obx * rby - oby * rbx;
        const float vrel_x = vcax - vcbx, vrel_y = vcay - vcby, vrel_z = vcaz - vcbz;
        const float vrel_n = vrel_x * nx + vrel_y * ny + vrel_z * nz;
        if (vrel_n < 0.f) {
            if (flags) *flags |= kSfNormal;
            const float j_n = __fdiv_rn(-vrel_n, w_total);
            float doa_x, doa_y, doa_z, dob_x, dob_y, dob_z;
            world_inv_inertia(B, ia, raxnx, raxny, raxnz, doa_x, doa_y, doa_z);
            world_inv_inertia(B, ib, rbxnx, rbxny, rbxnz, dob_x, dob_y, dob_z);
            if (wa != 0.f) {
                B.vx(ia) += wa * j_n * nx; B.vy(ia) += wa * j_n * ny; B.vz(ia) += wa * j_n * nz;
                B.wx(ia) += j_n * doa_x; B.wy(ia) += j_n * doa_y; B.wz(ia) += j_n * doa_z;
            }
            if (wb != 0.f) {
                B.vx(ib) -= wb * j_n * nx; B.vy(ib) -= wb * j_n * ny; B.vz(ib) -= wb * j_n * nz;
                B.wx(ib) -= j_n * dob_x; B.wy(ib) -= j_n * dob_y; B.wz(ib) -= j_n * dob_z;
            }
        }
    }
    if (mu > 0.f) {
        const float oax2 = B.wx(ia), oay2 = B.wy(ia), oaz2 = B.wz(ia);
        const float obx2 = B.wx(ib), oby2 = B.wy(ib), obz2 = B.wz(ib);
        const float vcax2 = B.vx(ia) + oay2 * raz - oaz2 * ray;
        const float vcay2 = B.vy(ia) + oaz2 * rax - oax2 * raz;
        const float vcaz2 = B.vz(ia) + oax2 * ray - oay2 * rax;
        const float vcbx2 = B.vx(ib) + oby2 * rbz - obz2 * rby;
        const float vcby2 = B.vy(ib) + obz2 * rbx - obx2 * rbz;
        const float vcbz2 = B.vz(ib) + obx2 * rby - oby2 * rbx;
        const float rvx = vcax2 - vcbx2, rvy = vcay2 - vcby2, rvz = vcaz2 - vcbz2;
        const float rvn = rvx * nx + rvy * ny + rvz * nz;
        const float vt_x = rvx - rvn * nx, vt_y = rvy - rvn * ny, vt_z = rvz - rvn * nz;
        const float vt2 = vt_x * vt_x + vt_y * vt_y + vt_z * vt_z;
        if (vt2 > 1e-12f) {
            const float vt_len = __fsqrt_rn(vt2);
            const float tx = __fdiv_rn(vt_x, vt_len), ty = __fdiv_rn(vt_y, vt_len), tz = __fdiv_rn(vt_z, vt_len);
            const float ratx = ray * tz - raz * ty, raty = raz * tx - rax * tz, ratz = rax * ty - ray * tx;
            const float rbtx = rby * tz - rbz * ty, rbty = rbz * tx - rbx * tz, rbtz = rbx * ty - rby * tx;
            float fIa_x, fIa_y, fIa_z, fIb_x, fIb_y, fIb_z;
            world_inv_inertia(B, ia, ratx, raty, ratz, fIa_x, fIa_y, fIa_z);
            world_inv_inertia(B, ib, rbtx, rbty, rbtz, fIb_x, fIb_y, fIb_z);
            const float wt = wa + wb + ratx * fIa_x + raty * fIa_y + ratz * fIa_z + rbtx * fIb_x + rbty * fIb_y +
                             rbtz * fIb_z;
            if (wt > 1e-10f) {
                const float j_n_static = __fdiv_rn(lc, dt * w_total);
                float j_t = __fdiv_rn(vt_len, wt);
                if (flags) *flags |= kSfFriction | (mu * j_n_static < j_t ? kSfClamped : 0u);
                j_t = fminf(j_t, mu * j_n_static);
                if (wa != 0.f) {
                    B.vx(ia) -= wa * j_t * tx; B.vy(ia) -= wa * j_t * ty; B.vz(ia) -= wa * j_t * tz;
                    B.wx(ia) -= j_t * fIa_x; B.wy(ia) -= j_t * fIa_y; B.wz(ia) -= j_t * fIa_z;
                }
                if (wb != 0.f) {
                    B.vx(ib) += wb * j_t * tx; B.vy(ib) += wb * j_t * ty; B.vz(ib) += wb * j_t * tz;
                    B.wx(ib) += j_t * fIb_x; B.wy(ib) += j_t * fIb_y; B.wz(ib) += j_t * fIb_z;
                }
            }
        }
    }
    return kSolveDone;
}

}  // namespace dyph

namespace dyph {

// ── one contact on two lanes ────────────────────────────────────────────────
// Contact solves wait for one another in long chains of few contacts each, so
// a solve's latency counts and lanes are idle. solve_contact's work is the same
// on its two bodies up to sign, with a few scalars of both in between: lane
// pair (2 i, 2 i + 1) takes contact i, each lane one body held in registers,
// and the scalars cross by shuffles. Half the instructions per contact and no
// shared-memory round trip between its steps. Every float is computed by the
// same operations in the same order as in solve_contact (negating a factor or
// a summand is exact), so the results are bit-identical.
struct SideBody {
    float px, py, pz, qw, qx, qy, qz, vx, vy, vz, wx, wy, wz;
    float m, ixx, iyy, izz, ixy, ixz, iyz;
};

template <class Bodies>
__device__ __forceinline__ void store_side(const Bodies& B, uint32_t i, const SideBody& s) {
    B.px(i) = s.px; B.py(i) = s.py; B.pz(i) = s.pz;
    B.qw(i) = s.qw; B.qx(i) = s.qx; B.qy(i) = s.qy; B.qz(i) = s.qz;
    B.vx(i) = s.vx; B.vy(i) = s.vy; B.vz(i) = s.vz;
    B.wx(i) = s.wx; B.wy(i) = s.wy; B.wz(i) = s.wz;
}

// World rotation rows of the body and the world inverse inertia times a vector
// (world_inv_inertia).
struct SideRot {
    float R00, R01, R02, R10, R11, R12, R20, R21, R22;
};
__device__ __forceinline__ SideRot side_rot(const SideBody& b) {
    const float qw = b.qw, qx = b.qx, qy = b.qy, qz = b.qz;
    SideRot r;
    r.R00 = 1.f - 2.f * (qy * qy + qz * qz); r.R01 = 2.f * (qx * qy + qz * qw); r.R02 = 2.f * (qx * qz - qy * qw);
    r.R10 = 2.f * (qx * qy - qz * qw); r.R11 = 1.f - 2.f * (qx * qx + qz * qz); r.R12 = 2.f * (qy * qz + qx * qw);
    r.R20 = 2.f * (qx * qz + qy * qw); r.R21 = 2.f * (qy * qz - qx * qw); r.R22 = 1.f - 2.f * (qx * qx + qy * qy);
    return r;
}
__device__ __forceinline__ void side_inv_inertia(const SideRot& r, const SideBody& b, float vx, float vy, float vz,
                                                 float& ox, float& oy, float& oz) {
    const float lx = r.R00 * vx + r.R10 * vy + r.R20 * vz;
    const float ly = r.R01 * vx + r.R11 * vy + r.R21 * vz;
    const float lz = r.R02 * vx + r.R12 * vy + r.R22 * vz;
    const float ilx = b.ixx * lx + b.ixy * ly + b.ixz * lz;
    const float ily = b.ixy * lx + b.iyy * ly + b.iyz * lz;
    const float ilz = b.ixz * lx + b.iyz * ly + b.izz * lz;
    ox = r.R00 * ilx + r.R01 * ily + r.R02 * ilz;
    oy = r.R10 * ilx + r.R11 * ily + r.R12 * ilz;
    oz = r.R20 * ilx + r.R21 * ily + r.R22 * ilz;
}

// The other lane's value, and a pair's (body a's, body b's) values.
__device__ __forceinline__ float other_side(float x) { return __shfl_xor_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ void both_sides(bool is_b, float mine, float& a, float& b) {
    const float o = other_side(mine);
    a = is_b ? o : mine;
    b = is_b ? mine : o;
}

// solve_contact by lane pairs: `is_b` lanes hold body b in S, the others body
// a. The whole warp calls it; pairs with `valid` false do nothing. Both lanes
// of a pair return the same code, lambda and flags. kAhead takes the quotients
// by w_total together before the position correction (the relative velocity
// needs none of it): a shorter chain for more work, for callers that latency
// bounds.
template <bool kAhead = false>
__device__ __forceinline__ int solve_contact_side(bool valid, bool is_b, SideBody& S, const Contact& ct, float mu,
                                                  float& lc, float dt, uint32_t* flags = nullptr) {
    constexpr unsigned kAll = 0xffffffffu;
    const float depth = ct.depth;
    const float remaining = depth - lc;
    const bool wanted = valid && !(depth <= 0.f) && !(remaining <= 1e-6f);
    if (!__any_sync(kAll, wanted)) return kSolveSkipped;
    const float nx = ct.nx, ny = ct.ny, nz = ct.nz;
    const float m = S.m, ms = is_b ? -m : m;  // the impulse acts with opposite signs
    const bool dynamic = m != 0.f;
    const float rx = ct.px - S.px, ry = ct.py - S.py, rz = ct.pz - S.pz;
    const float rnx = ry * nz - rz * ny, rny = rz * nx - rx * nz, rnz = rx * ny - ry * nx;
    float ix, iy, iz;
    side_inv_inertia(side_rot(S), S, rnx, rny, rnz, ix, iy, iz);
    float wa, wb, wa_ang, wb_ang;
    both_sides(is_b, m, wa, wb);
    both_sides(is_b, rnx * ix + rny * iy + rnz * iz, wa_ang, wb_ang);
    const float w_total = wa + wb + wa_ang + wb_ang;
    const bool act = wanted && !(w_total < 1e-10f);
    uint32_t fl = act ? kSfActive : 0u;
    // contact velocities of a minus b along the normal
    auto normal_velocity = [&]() {
        float vax, vbx, vay, vby, vaz, vbz;
        both_sides(is_b, S.vx + S.wy * rz - S.wz * ry, vax, vbx);
        both_sides(is_b, S.vy + S.wz * rx - S.wx * rz, vay, vby);
        both_sides(is_b, S.vz + S.wx * ry - S.wy * rx, vaz, vbz);
        return (vax - vbx) * nx + (vay - vby) * ny + (vaz - vbz) * nz;
    };
    float vrel_n = 0.f, dl = 0.f, j_n = 0.f, j_n_static = 0.f;
    if (kAhead) {
        vrel_n = normal_velocity();
        const float w_div = act ? w_total : 1.f;  // an idle pair divides by 1
        dl = __fdiv_rn(act ? remaining : 1.f, w_div);
        j_n = __fdiv_rn(act ? -vrel_n : 1.f, w_div);
        j_n_static = __fdiv_rn(act ? lc + remaining : 1.f, act ? dt * w_div : 1.f);
    }
    if (act) {
        if (!kAhead) dl = __fdiv_rn(remaining, w_total);
        lc += remaining;
        if (dynamic) {
            S.px += ms * dl * nx; S.py += ms * dl * ny; S.pz += ms * dl * nz;
            const float sdl = is_b ? -dl : dl;
            const float ax = sdl * ix, ay = sdl * iy, az = sdl * iz;
            const float qw = S.qw, qx = S.qx, qy = S.qy, qz = S.qz;
            S.qw += 0.5f * (-ax * qx - ay * qy - az * qz);
            S.qx += 0.5f * (ax * qw + ay * qz - az * qy);
            S.qy += 0.5f * (-ax * qz + ay * qw + az * qx);
            S.qz += 0.5f * (ax * qy - ay * qx + az * qw);
        }
    }
    const SideRot rot = side_rot(S);
    if (!kAhead) vrel_n = normal_velocity();
    if (act && vrel_n < 0.f) {
        fl |= kSfNormal;
        if (dynamic) {
            if (!kAhead) j_n = __fdiv_rn(-vrel_n, w_total);
            float dx, dy, dz;
            side_inv_inertia(rot, S, rnx, rny, rnz, dx, dy, dz);
            const float sj = is_b ? -j_n : j_n;
            S.vx += ms * j_n * nx; S.vy += ms * j_n * ny; S.vz += ms * j_n * nz;
            S.wx += sj * dx; S.wy += sj * dy; S.wz += sj * dz;
        }
    }
    if (mu > 0.f) {
        float vax, vbx, vay, vby, vaz, vbz;
        both_sides(is_b, S.vx + S.wy * rz - S.wz * ry, vax, vbx);
        both_sides(is_b, S.vy + S.wz * rx - S.wx * rz, vay, vby);
        both_sides(is_b, S.vz + S.wx * ry - S.wy * rx, vaz, vbz);
        const float rvx = vax - vbx, rvy = vay - vby, rvz = vaz - vbz;
        const float rvn = rvx * nx + rvy * ny + rvz * nz;
        const float vt_x = rvx - rvn * nx, vt_y = rvy - rvn * ny, vt_z = rvz - rvn * nz;
        const float vt2 = vt_x * vt_x + vt_y * vt_y + vt_z * vt_z;
        const bool slides = act && vt2 > 1e-12f;
        if (__any_sync(kAll, slides)) {
            float vt_len = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
            if (slides) {
                vt_len = __fsqrt_rn(vt2);
                tx = __fdiv_rn(vt_x, vt_len);
                ty = __fdiv_rn(vt_y, vt_len);
                tz = __fdiv_rn(vt_z, vt_len);
            }
            const float rtx = ry * tz - rz * ty, rty = rz * tx - rx * tz, rtz = rx * ty - ry * tx;
            float fx, fy, fz;
            side_inv_inertia(rot, S, rtx, rty, rtz, fx, fy, fz);
            float ax, bx, ay, by, az, bz;
            both_sides(is_b, rtx * fx, ax, bx);
            both_sides(is_b, rty * fy, ay, by);
            both_sides(is_b, rtz * fz, az, bz);
            const float wt = wa + wb + ax + ay + az + bx + by + bz;
            if (slides && wt > 1e-10f) {
                if (!kAhead) j_n_static = __fdiv_rn(lc, dt * w_total);
                float j_t = __fdiv_rn(vt_len, wt);
                fl |= kSfFriction | (mu * j_n_static < j_t ? kSfClamped : 0u);
                j_t = fminf(j_t, mu * j_n_static);
                if (dynamic) {
                    const float sj = is_b ? j_t : -j_t;
                    S.vx -= ms * j_t * tx; S.vy -= ms * j_t * ty; S.vz -= ms * j_t * tz;
                    S.wx += sj * fx; S.wy += sj * fy; S.wz += sj * fz;
                }
            }
        }
    }
    if (flags) *flags = fl;
    return act ? kSolveDone : (wanted ? kSolveDeferred : kSolveSkipped);
}

}  // namespace dyph
