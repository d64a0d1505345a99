// The uniform-grid step on sm_100a: face pass, update pass (positivity ratio, continuity, level lookup; in the device loop
// also the clocks and the next step's settings), the step's end (boundary cells, tally, lines, envelope), active-list
// rebuild; all of them in one kernel (the resident loop); and the layout converters.
//
// A CTA takes one 32 x 32 tile, or a strip of one, at a time, looping over its share of the work list (grid-stride, so a
// graph-captured launch serves any list length): the face pass with 512 threads (a thread a column, two rows; 256 or 128
// in its strip forms), the update pass with 256 (a thread a column, four rows). State sits in the dense NATIVE layout, so a neighbour is an address offset and
// the reference's halo exchanges (wadi2d/solver/gpu/kernels/cells.cu:80-93) disappear; the guard ring is zero like
// the reference's void tile. In a batch every tile reads its run's clock, cell size, flags and current half.
//
// The face pass restates wadi2d/solver/gpu/kernels/faces.cu:10-175 (= wadi2d/solver/cpu/kernels.py:86-244); the
// update pass fuses limit and update (cells.cu:4-63, kernels.py:247-299) by computing the positivity ratio r of the
// tile and its one-cell ring in shared memory; the step's end restates cells.cu:95-111 and engine/maxima.py:53-92.
#include <cstdio>

#include "w2b_common.cuh"
#include "w2b_loop.cuh"
#include "w2b_tma.cuh"

namespace w2b {

// The face and update passes are compiled twice (wadi2d_b200/build.py): into namespace exact with the library's IEEE
// flags, the reference's float32 bits, and into namespace fast with W2B_FAST and FMA contraction (the approximate
// division, square root and cube root and the hardware max and min of w2b_common.cuh qdiv/qsqrt/qcbrt/qmax/qmin, in
// the face arithmetic). W2BParams.arith picks one per handle.
// Everything after them (envelope, boundary, control, converters) is compiled once, with the exact build.
#ifdef W2B_FAST
#define W2B_ARITH fast
#else
#define W2B_ARITH exact
#endif
namespace W2B_ARITH {

// ------------------------------------------------------------------ face pass

// Shared-memory image of one tile for the face pass. Boxes of 40 x 36 floats hold the tile with 2 cells of halo north
// and south and 4 west and east (the TMA box starts on a 16-byte boundary); own cell (j, i) sits at box (j + 2, i + 4).
constexpr int BOXW = 40, BOXH = 36, BOX = BOXW * BOXH;
constexpr int F_D = 0, F_H = 1, F_U = 2, F_V = 3, F_QX = 4, F_QY = 5, F_OM = 6, F_ZCX = 7, F_ZCY = 8, NBOX = 9;
constexpr int SM_M = NBOX * BOX;          // mx, my: 32 x 32 each
constexpr int SM_ST = SM_M + 2 * TILE2;   // the 12 static face scalars of the tile, 32 x 32 each
constexpr int SM_FLOATS = SM_ST + 12 * TILE2;
constexpr int FACES_SMEM = SM_FLOATS * 4;  // 109,184 bytes: two CTAs a SM
constexpr int FACES_THREADS = 512;

// The two images the face helpers read. off(f) is the offset of state field f's array as the helpers index it, by
// box index b (b's row 0 is two rows above the tile's or strip's first row, its column 0 four columns west of the
// first column; a row is BOXW floats). A whole tile (the face pass and the probe): nine 40 x 36 boxes, the plan share
// among them. A strip (the strip forms of the face pass): each state field's box holds only the rows the face
// arithmetic reads, the plan share is read from global memory on the refresh steps that want it. S is the stride of a
// static face scalar's (and of a momentum's) array in the image: 1,024 floats for a tile, 32 H for a strip.
struct TileImage {
    static constexpr int M = SM_M, ST = SM_ST, S = TILE2;
    static constexpr int HO = SM_M;  // the last step's mean depth box (40 x 36), in the momenta's place
    static constexpr bool OM = true;
    __host__ __device__ static constexpr int off(int f) { return f * BOX; }
};
__host__ __device__ constexpr int pad32(int n) { return (n + 31) / 32 * 32; }  // floats, to a 128-byte boundary
template <int H>
struct StripImage {
    // The rows of each field's box around a strip of H rows, from the face arithmetic's reads (b - S, b, b + S,
    // b +- 2 S, b +- PP, b +- 2 PP of face_in, face_a, face_bc): the velocities two rows above to two below; depth,
    // mean depth, x discharge and the y lip one row above to the last row; the y discharge one above to one below;
    // the x lip the strip's own rows.
    static constexpr int R_UV = H + 4, R_QY = H + 2, R_ZCX = H, R_1 = H + 1;
    // each box's region, 128-byte aligned, in the order u v d h qx qy zcx zcy (u first: every offset is >= 0)
    static constexpr int S_U = 0, S_V = S_U + pad32(BOXW * R_UV), S_D = S_V + pad32(BOXW * R_UV);
    static constexpr int S_H = S_D + pad32(BOXW * R_1), S_QX = S_H + pad32(BOXW * R_1);
    static constexpr int S_QY = S_QX + pad32(BOXW * R_1), S_ZCX = S_QY + pad32(BOXW * R_QY);
    static constexpr int S_ZCY = S_ZCX + pad32(BOXW * R_ZCX), S_END = S_ZCY + pad32(BOXW * R_1);
    static constexpr int M = S_END, ST = S_END + 2 * TILE * H, S = TILE * H;
    // the last step's mean depth box, in the momenta's place: the rows of the mean depth's box, BOXW * (H + 1) <=
    // 2 TILE H floats
    static constexpr int HO = M - BOXW;
    static constexpr bool OM = false;
    static constexpr int FLOATS = ST + 12 * S;
    static constexpr int SMEM = FLOATS * 4;        // 51,840 bytes for 16 rows (four CTAs a SM), 27,264 for 8 (eight)
    // the bytes the strip's copies bring (the regions without their padding): with the momenta, or with the last
    // step's mean depth in their place
    static constexpr int BYTES = 4 * (BOXW * (2 * R_UV + 4 * R_1 + R_QY + R_ZCX) + 14 * TILE * H);
    static constexpr int BYTES_HO = BYTES - 4 * (2 * TILE * H - BOXW * R_1);
    static constexpr int THREADS = 16 * H;         // a warp two rows
    static constexpr int CTAS = H == 16 ? 4 : 8;   // resident CTAs a SM the launch bound plans for
    __host__ __device__ static constexpr int off(int f) {
        return f == F_U   ? S_U
             : f == F_V   ? S_V
             : f == F_D   ? S_D - BOXW
             : f == F_H   ? S_H - BOXW
             : f == F_QX  ? S_QX - BOXW
             : f == F_QY  ? S_QY - BOXW
             : f == F_ZCX ? S_ZCX - 2 * BOXW
                          : S_ZCY - BOXW;
    }
};
static_assert(StripImage<8>::SMEM == 27264 && StripImage<16>::SMEM == 51840, "strip image sizes");
static_assert(StripImage<8>::off(F_D) >= 0 && StripImage<8>::off(F_ZCX) >= 0, "strip offsets");
static_assert(BOXW * StripImage<8>::R_1 <= 2 * TILE * 8 && BOXW * StripImage<16>::R_1 <= 2 * TILE * 16 &&
                  BOX <= 2 * TILE2,
              "the last step's mean depth box fits the momenta's place");

// What the first part of a face hands to the rest: the row's quad (its load is issued in part A and consumed after
// the table-free momentum terms), the face depth, and the table row with the upwind choice, the live flag and the
// above-the-table flag packed in one word. Parts B and C re-read the other inputs from the tile's image, so few
// registers stay live across the momentum terms.
struct FaceA {
    float4 q;
    float eface;
    int bits;
};
constexpr int FA_ROW = 0xff, FA_LEFT = 0x100, FA_LIVE = 0x200, FA_ABOVE = 0x400;

// The face's upwind inputs from the tile's image (wadi2d/solver/gpu/kernels/faces.cu:19-31): the levels over each
// side's invert, their positive parts, and the velocity on the face.
struct FaceIn {
    float e_l, e_r, e_lp, e_rp, uf;
};
template <int AX, class L>
__device__ __forceinline__ FaceIn face_in(const float* sm, int b, int sl) {
    constexpr int S = AX == 0 ? 1 : BOXW;
    const float* D = sm + L::off(F_D);
    const float* U = sm + L::off(AX == 0 ? F_U : F_V);
    const float* st = sm + L::ST + AX * 6 * L::S;
    FaceIn I;
    I.e_l = D[b - S] - st[0 * L::S + sl];
    I.e_r = D[b] - st[1 * L::S + sl];
    I.uf = U[b];
    I.e_lp = qmax(I.e_l, 0.0f);
    I.e_rp = qmax(I.e_r, 0.0f);
    return I;
}

// Part A of the face of axis AX at box index b (wadi2d/solver/gpu/kernels/faces.cu:19-44).
// ON: the numerics switches (second-order momentum, sheet flow, dry-face mirroring, depth carry) are all on, as the
// reference's defaults have them, and known to the compiler; otherwise they are read from A.P.
// L: the image (TileImage, StripImage); sl: the cell's index in the image's static arrays, local: in the tile.
template <int AX, bool ON = false, class L = TileImage>
__device__ __forceinline__ void face_a(const float* sm, int b, int sl, int local, const StepArgs& A, int t,
                                       FaceA& F) {
    constexpr int S = AX == 0 ? 1 : BOXW;
    const W2BParams& P = A.P;
    const float* st = sm + L::ST + AX * 6 * L::S;
    const FaceIn I = face_in<AX, L>(sm, b, sl);
    const bool from_left = I.uf > 0.0f || (I.uf == 0.0f && I.e_l >= I.e_r);
    const float eup = from_left ? I.e_lp : I.e_rp;
    F.bits = from_left ? FA_LEFT : 0;
    if (eup <= P.e_wet) return;
    const float cwf = st[5 * L::S + sl];
    const float top = st[4 * L::S + sl];
    float eface = eup;
    if ((ON || P.carry) && cwf == 0.0f) {
        const float* ZC = sm + L::off(AX == 0 ? F_ZCX : F_ZCY);
        const float dz = from_left ? ZC[b - S] - st[0 * L::S + sl] : ZC[b] - st[1 * L::S + sl];
        if (dz > 1e-6f) {
            float phi = qdiv(eup - 2.0f * dz, 2.0f * dz);
            phi = phi < 0.0f ? 0.0f : (phi > 1.0f ? 1.0f : phi);
            eface = eup - phi * dz;
        }
    }
    const int last = A.rows - 1;
    const bool above = eface >= top;
    const int r = above ? last - 1 : row_of(qsqrt(qdiv(eface, top)) * (float)last, last);
    F.eface = eface;
    F.bits |= FA_LIVE | (above ? FA_ABOVE : 0) | r;
    const float4* quads = A.ftab4[AX] + (size_t)t * (A.rows - 1) * TILE2 + local;
    F.q = __ldg(quads + (size_t)r * TILE2);
}

// Parts B and C: the momentum terms (faces.cu:50-100, table-free), then the lookup, section, friction, crest cap,
// outputs and wave speed (faces.cu:43-44, :52-63, :102-145). Returns the wave speed.
// mst: the face's momentum is the image's stored one (Ctl::m_stored), else it is formed from the last step's mean
// depths (the image's HO box) and the face velocity, as the step that wrote the velocity formed it. The new momentum
// is not written: the next step forms it the same way.
// PROBE: write the face's new velocity to probe_un[local] and nothing of the state (the step-limiter probe).
template <int AX, bool PROBE = false, bool ON = false, class L = TileImage>
__device__ __forceinline__ float face_bc(const float* sm, int b, int sl, int local, int k, const StepArgs& A, int t,
                                         const FaceA& F, float dt, float dx, int want_wave, const float* rowc, int p,
                                         int mst, float* probe_un = nullptr) {
    constexpr int S = AX == 0 ? 1 : BOXW;
    constexpr int PP = AX == 0 ? BOXW : 1;
    const W2BParams& P = A.P;
    if (!(F.bits & FA_LIVE)) {
        if constexpr (PROBE) {
            probe_un[local] = 0.0f;
        } else {
            A.uu[AX][1 - p][k] = 0.0f;
            A.q1[AX][k] = 0.0f;
        }
        return 0.0f;
    }
    const float ZERO = 0.0f, HALF = 0.5f, ONE = 1.0f;
    const float span = dx;
    const float* H = sm + L::off(F_H);
    const float* U = sm + L::off(AX == 0 ? F_U : F_V);
    const float* VP = sm + L::off(AX == 0 ? F_V : F_U);
    const float* Q = sm + L::off(AX == 0 ? F_QX : F_QY);
    const float* QP = sm + L::off(AX == 0 ? F_QY : F_QX);
    const float* st = sm + L::ST + AX * 6 * L::S;
    const FaceIn I = face_in<AX, L>(sm, b, sl);
    const bool from_left = (F.bits & FA_LEFT) != 0;
    const float uf = I.uf;
    const float eup = from_left ? I.e_lp : I.e_rp;
    const float h_l = H[b - S], h_r = H[b];
    const float hup = from_left ? h_l : h_r;

    // [1] section: the disconnected drive (the volume-limited section needs the table, below)
    float d_eta = I.e_rp - I.e_lp;
    if (ON || P.sheet) {
        const float edown = from_left ? I.e_rp : I.e_lp;
        if (edown <= ZERO) {
            const float g_u = from_left ? st[2 * L::S + sl] : st[3 * L::S + sl];
            const float g_d = from_left ? st[3 * L::S + sl] : st[2 * L::S + sl];
            const float h_d = from_left ? h_r : h_l;
            const float drop = (hup - g_u) - qmax(h_d - g_d, HALF * (g_u - g_d));
            const float level_drop = fabsf(I.e_l - I.e_r);
            const float drive = qmax(eup, qmin(drop, level_drop));
            d_eta = from_left ? -drive : drive;
        }
    }
    // [3] momentum fluxes
    const int mirror = ON ? 1 : P.mirror, second = ON ? 1 : P.second;
    const float um = gated(U[b - S], uf, mirror);
    const float up = gated(U[b + S], uf, mirror);
    const float umm = gated(U[b - 2 * S], um, mirror);
    const float upp = gated(U[b + 2 * S], up, mirror);
    const float qk = Q[b];
    const float qc_l = HALF * (Q[b - S] + qk);
    const float qc_r = HALF * (qk + Q[b + S]);
    // each upwind choice picks the arguments of one ustar (the same value as choosing between two ustar calls)
    const bool pl = qc_l > ZERO, pr = qc_r > ZERO;
    const float s_l = ustar(pl ? um : uf, pl ? umm : up, pl ? uf : um, second);
    const float s_r = ustar(pr ? uf : up, pr ? um : upp, pr ? up : uf, second);
    float flux = qc_r * s_r - qc_l * s_l;
    const float qy_s = HALF * (QP[b - S] + QP[b]);
    const float qy_n = HALF * (QP[b - S + PP] + QP[b + PP]);
    const float u_s = gated(U[b - PP], uf, mirror);
    const float u_n = gated(U[b + PP], uf, mirror);
    const float uss = gated(U[b - 2 * PP], u_s, mirror);
    const float unn = gated(U[b + 2 * PP], u_n, mirror);
    const bool ps = qy_s > ZERO, pn = qy_n > ZERO;
    const float us_s = ustar(ps ? u_s : uf, ps ? uss : u_n, ps ? uf : u_s, second);
    const float us_n = ustar(pn ? uf : u_n, pn ? u_s : unn, pn ? u_n : uf, second);
    flux += qy_n * us_n - qy_s * us_s;
    // [4] momentum and pressure (the fast build multiplies by one reciprocal of the span, which the compiler hoists
    // out of the tile's loop)
    const float abar = HALF * (h_l + h_r) * dx;
    // the face's momentum (the last step's abar * u, rounded once as that step rounded it)
    const float* HO = sm + L::HO;
    auto momentum = [&]() {
        return mst ? sm[L::M + AX * L::S + sl] : __fmul_rn(HALF * (HO[b - S] + HO[b]) * dx, uf);
    };
#ifdef W2B_FAST
    const float rspan = rcp_approx(span);
    const float press = dt * P.g * d_eta * rspan;
    float us;
    if (abar > 1e-6f * dx)
        us = qdiv(momentum() - dt * flux * rspan, abar) - press;
    else
        us = uf - press;
#else
    const float press = qdiv(dt * P.g * d_eta, span);
    float us;
    if (abar > 1e-6f * dx)
        us = qdiv(momentum() - qdiv(dt * flux, span), abar) - press;
    else
        us = uf - press;
#endif
    const float vb = 0.25f * (VP[b - S] + VP[b] + VP[b - S + PP] + VP[b + PP]);

    // the table lookup from the quad loaded in part A (common.cuh face_lookup); rowc holds, per row r, c0^2 and
    // c1^2 - c0^2 with c0 = r / m, c1 = (r + 1) / m, and in its last slot 1 - c^2 with c = (m - 1) / m: the very
    // float32 values the lookup forms, computed once a CTA
    const float top = st[4 * L::S + sl], e = F.eface;
    const float4 q = F.q;
    float area, tt, w;
    if (F.bits & FA_ABOVE) {
        const float a1 = q.z, a0 = q.x;
        w = qdiv(a1 - a0, top * rowc[2 * (A.rows - 1)]);
        area = a1 + w * (e - top);
        tt = q.w * qdiv(area, qmax(a1, 1e-12f));
    } else {
        const int r = F.bits & FA_ROW;
        const float e0 = rowc[2 * r] * top;
        const float de = rowc[2 * r + 1] * top;
#ifdef W2B_FAST
        const float rde = rcp_approx(de);  // one reciprocal for both quotients
        const float f = (e - e0) * rde;
        area = q.x + f * (q.z - q.x);
        tt = q.y + f * (q.w - q.y);
        w = (q.z - q.x) * rde;
#else
        const float f = qdiv(e - e0, de);
        area = q.x + f * (q.z - q.x);
        tt = q.y + f * (q.w - q.y);
        w = qdiv(q.z - q.x, de);
#endif
    }
    // [1] the volume-limited section
    float rho = ONE;
    if (ON || P.sheet) {
        const float avol = hup * dx;
        if (avol < area) {
            const float sub = qdiv(qmin(I.e_lp, I.e_rp), qmax(I.e_lp, I.e_rp));
            const float sub2 = sub * sub;
            const float alpha = sub2 * sub2;
            rho = alpha + qdiv((ONE - alpha) * avol, area);
        }
    }
    // [5] friction. The fast build forms 1 / max(tt^(10/3), 1e-30) and 1 / max(rho^(4/3), 1e-12) as capped powers from
    // the hardware log2 and exp2 (within about 1e-6 relative; tt = 0 or rho = 0 gives the cap, as the clamps do).
#ifdef W2B_FAST
    float fric = area * area * qmin(ex2_approx(-3.33333325f * lg2_approx(tt)), 1e30f);
    if (rho < ONE) fric = fric * qmin(ex2_approx(-1.33333337f * lg2_approx(rho)), 1e12f);
#else
    const float t3 = tt * tt * tt * qcbrt(tt);
    float fric = qdiv(area * area, qmax(t3, 1e-30f));
    if (rho < ONE) fric = qdiv(fric, qmax(rho * qcbrt(rho), 1e-12f));
#endif
    const float a = dt * P.g * fric;
    const float sp = qsqrt(us * us + vb * vb);
    float un = qdiv(2.0f * us, ONE + qsqrt(ONE + 4.0f * a * sp));
    if (fabsf(un) > P.u_max) un = un > ZERO ? P.u_max : -P.u_max;
    // [6] crest face
    float qn = area * rho * un;
    float c = st[5 * L::S + sl];
    if (c != ZERO) {
        float area_c = area, w_c = w;
        if (c < ZERO) {
            c = -c;
            const float ua = from_left ? um : up;
            float tc;
            const float4* quads = A.ftab4[AX] + (size_t)t * (A.rows - 1) * TILE2 + local;
            face_lookup(eup + qdiv(HALF * ua * ua, P.g), top, quads, A.rows, area_c, tc, w_c);
        }
        const float qc = c * area_c * qsqrt(qdiv(area_c, qmax(w_c, 1e-9f)));
        if (fabsf(qn) > qc) {
            qn = qn > ZERO ? qc : -qc;
            un = qdiv(qn, qmax(area * rho, 1e-12f));
        }
    }
    if constexpr (PROBE) {
        probe_un[local] = un;
    } else {
        A.uu[AX][1 - p][k] = un;
        A.q1[AX][k] = qn;
    }
    if (!want_wave) return ZERO;
    if (not_finite(un)) return 1e30f;
    const float* D = sm + L::off(F_D);
    const float d_left = D[b - S], d_right = D[b];
    const float dup = from_left ? d_left : d_right;
    if (dup <= P.h_cfl) return ZERO;
    // the plan shares of the face's two cells: from the image, or (a strip) from global memory at native index k
    float om_l, om_r;
    if constexpr (L::OM) {
        const float* OM = sm + L::off(F_OM);
        om_l = OM[b - S];
        om_r = OM[b];
    } else {
        om_l = A.om[k - (AX == 0 ? 1 : A.px)];
        om_r = A.om[k];
    }
    float plan = from_left ? om_l : om_r;
    const float dother = from_left ? d_right : d_left;
    if (dother > P.h_cfl) plan = qmin(plan, from_left ? om_r : om_l);
    const float wave = qsqrt(qmax(qdiv(P.g * area * rho, qmax(plan, P.a_min) * dx), ZERO));
    return fabsf(un) + qmin(P.lead * fabsf(un - uf), 2.0f * wave) + wave;
}

__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax32(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide max of v; the result is valid in thread 0. red holds one entry a warp.
__device__ __forceinline__ float block_max(float v, float* red) {
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int nw = (int)(blockDim.x * blockDim.y) / 32;
    v = warp_max(v);
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    float r = 0.0f;
    if (tid < 32) {
        r = tid < nw ? red[tid] : 0.0f;
        r = warp_max(r);
    }
    __syncthreads();
    return r;
}

// Threads' part of a table of the row constants that the table lookup forms (face_bc's rowc), one a CTA.
__device__ __forceinline__ void fill_rowc(float* rowc, int rows) {
    const int tid = threadIdx.x;
    if (tid < rows - 1) {
        const float m = (float)(rows - 1);
        const float c0 = (float)tid / m;
        const float c1 = (float)(tid + 1) / m;
        rowc[2 * tid] = c0 * c0;
        rowc[2 * tid + 1] = c1 * c1 - c0 * c0;
    } else if (tid == rows - 1) {
        const float m = (float)(rows - 1);
        const float c = (m - 1.0f) / m;
        rowc[2 * tid] = 1.0f - c * c;
    }
}

// The face pass: both own faces of every cell of the tiles of the work list (wadi2d/solver/gpu/kernels/faces.cu:
// 148-175). Each CTA (16 warps, a warp a tile row, two rows a warp; two CTAs a SM) stages a tile with TMA: nine
// 40 x 36 state boxes, the two momenta (or, once a face pass has stepped, the last step's mean depth box they are
// formed from), and the tile's twelve static face scalars as bulk copies; on refresh steps
// the tile's wave maximum goes to its run's maximum (an integer atomic max on the float bits). p is the parity of
// the run's ping-pong halves.
template <bool ON>
__global__ void __launch_bounds__(FACES_THREADS, 2) faces_kernel(const __grid_constant__ TileMaps M, StepArgs A) {
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ float red[32];
    __shared__ float rowc[2 * 64 + 1];
    Ctl* ctl = A.ctl;
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    fill_rowc(rowc, A.rows);
    __syncthreads();
    if (!(*A.any & ANY_RUN)) return;
    const int nwork = ctl->nwork;
    const int mst = ctl->m_stored;
    const float* statics[12] = {A.fl[0], A.fr[0], A.gl[0], A.gr[0], A.ef[0], A.cw[0],
                                A.fl[1], A.fr[1], A.gl[1], A.gr[1], A.ef[1], A.cw[1]};
    uint32_t phase = 0;
    const int lane = tid & 31, warp = tid >> 5;
    for (int a = blockIdx.x; a < nwork; a += gridDim.x) {
        const int t = A.list[a];
        const int run = A.tile_run[t];
        const int flags = A.R.flags[run];
        if (!(flags & F_RUN)) continue;  // the tile's run has finished: uniform over the CTA
        const float dt = A.R.dtf[run];
        const float dx = A.R.dx[run];
        const int want_wave = (flags & F_WAVE) != 0;
        const int p = A.R.parity[run];
        const int tj = A.tiles[2 * t], ti = A.tiles[2 * t + 1];
        const int ts = table_of(A, t);
        if (tid == 0) {
            fence_proxy_async();
            mbar_expect_tx(&bar, (uint32_t)((NBOX - (want_wave ? 0 : 1)) * BOX + (mst ? 14 * TILE2 : BOX + 12 * TILE2)) * 4u);
            const int x0 = ti * TILE + GX - 4, y0 = tj * TILE + GY - 2;
            tma_load_2d(sm + F_D * BOX, &M.d, x0, y0, &bar);
            tma_load_2d(sm + F_H * BOX, &M.h[p], x0, y0, &bar);
            tma_load_2d(sm + F_U * BOX, &M.u[p], x0, y0, &bar);
            tma_load_2d(sm + F_V * BOX, &M.v[p], x0, y0, &bar);
            tma_load_2d(sm + F_QX * BOX, &M.qx, x0, y0, &bar);
            tma_load_2d(sm + F_QY * BOX, &M.qy, x0, y0, &bar);
            if (want_wave) tma_load_2d(sm + F_OM * BOX, &M.om, x0, y0, &bar);
            tma_load_2d(sm + F_ZCX * BOX, &M.zcx, x0, y0, &bar);
            tma_load_2d(sm + F_ZCY * BOX, &M.zcy, x0, y0, &bar);
            if (mst) {
                tma_load_2d(sm + SM_M, &M.mx[p], x0 + 4, y0 + 2, &bar);
                tma_load_2d(sm + SM_M + TILE2, &M.my[p], x0 + 4, y0 + 2, &bar);
            } else {
                tma_load_2d(sm + TileImage::HO, &M.h[1 - p], x0, y0, &bar);
            }
            for (int f = 0; f < 12; ++f) bulk_load(sm + SM_ST + f * TILE2, statics[f] + (size_t)ts * TILE2, TILE2 * 4, &bar);
        }
        const bool ok = mbar_wait(&bar, phase);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            // the copies did not land: report, give them one more bounded wait, and leave the loop
            if (tid == 0) atomicExch(&ctl->status, W2B_ETIMEOUT);
            mbar_wait(&bar, phase ^ 1u);
            return;
        }
        const int base = (tj * TILE + GY) * A.px + ti * TILE + GX;
        float wmax = 0.0f;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            const int jj = warp + 16 * c, ii = lane;
            const int local = jj * TILE + ii;
            const int b = (jj + 2) * BOXW + ii + 4;
            const int k = base + jj * A.px + ii;
            FaceA fx, fy;
            face_a<0, ON>(sm, b, local, local, A, ts, fx);
            face_a<1, ON>(sm, b, local, local, A, ts, fy);
            const float wx = face_bc<0, false, ON>(sm, b, local, local, k, A, ts, fx, dt, dx, want_wave, rowc, p, mst);
            const float wy = face_bc<1, false, ON>(sm, b, local, local, k, A, ts, fy, dt, dx, want_wave, rowc, p, mst);
            wmax = fmax32(wmax, fmax32(wx, wy));
        }
        if (want_wave) {
            // the tile's wave, and the run's maximum (wadi2d/solver/gpu/kernels/common.cuh:93-96: positive floats
            // order like their bit patterns, so the integer maximum is the float maximum)
            const float bm = block_max(wmax, red);
            if (tid == 0) {
                A.wave[t] = bm;
                atomicMax(A.R.wave_bits + run, __float_as_uint(bm));
            }
        } else {
            __syncthreads();
        }
    }
}

// The wave speed and the new velocity of every own face of tile t for a step dt from the current state, as the face
// pass would compute them, written to out ([wx | wy | un_x | un_y], 1024 each, tile layout) and nothing else: the
// device side of the step limiter (wadi2d/solver/limiter.py:31-55, the CPU twin's face_step on one tile). One CTA;
// the tile's image is filled with plain loads (the boxes lie inside the guard ring of the NATIVE arrays).
__global__ void __launch_bounds__(1024) probe_kernel(StepArgs A, int t, float dt, float* __restrict__ out) {
    extern __shared__ __align__(128) float sm[];
    __shared__ float rowc[2 * 64 + 1];
    const int tid = threadIdx.x;
    const int run = A.tile_run[t];
    const int p = A.R.parity[run];
    const float dx = A.R.dx[run];
    const int tj = A.tiles[2 * t], ti = A.tiles[2 * t + 1];
    const int x0 = ti * TILE + GX - 4, y0 = tj * TILE + GY - 2;
    const int mst = A.ctl->m_stored;
    const float* boxes[NBOX] = {A.d, A.hh[p], A.uu[0][p], A.uu[1][p], A.q[0], A.q[1], A.om, A.zc[0], A.zc[1]};
    for (int idx = tid; idx < BOX; idx += blockDim.x) {
        const size_t k = (size_t)(y0 + idx / BOXW) * A.px + x0 + idx % BOXW;
        for (int f = 0; f < NBOX; ++f) sm[f * BOX + idx] = boxes[f][k];
        if (!mst) sm[TileImage::HO + idx] = A.hh[1 - p][k];
    }
    const float* statics[12] = {A.fl[0], A.fr[0], A.gl[0], A.gr[0], A.ef[0], A.cw[0],
                                A.fl[1], A.fr[1], A.gl[1], A.gr[1], A.ef[1], A.cw[1]};
    for (int idx = tid; idx < TILE2; idx += blockDim.x) {
        const size_t k = (size_t)(tj * TILE + GY + idx / TILE) * A.px + ti * TILE + GX + idx % TILE;
        if (mst) {
            sm[SM_M + idx] = A.mm[0][p][k];
            sm[SM_M + TILE2 + idx] = A.mm[1][p][k];
        }
        for (int f = 0; f < 12; ++f) sm[SM_ST + f * TILE2 + idx] = statics[f][(size_t)table_of(A, t) * TILE2 + idx];
    }
    fill_rowc(rowc, A.rows);
    __syncthreads();
    const int jj = tid >> 5, ii = tid & 31;
    const int local = jj * TILE + ii;
    const int b = (jj + 2) * BOXW + ii + 4;
    const int k = (tj * TILE + GY + jj) * A.px + ti * TILE + GX + ii;
    FaceA fx, fy;
    const int ts = table_of(A, t);
    face_a<0>(sm, b, local, local, A, ts, fx);
    face_a<1>(sm, b, local, local, A, ts, fy);
    out[local] = face_bc<0, true>(sm, b, local, local, k, A, ts, fx, dt, dx, 1, rowc, p, mst, out + 2 * TILE2);
    out[TILE2 + local] = face_bc<1, true>(sm, b, local, local, k, A, ts, fy, dt, dx, 1, rowc, p, mst, out + 3 * TILE2);
}

void launch_probe(const StepArgs& A, int t, float dt, float* out, cudaStream_t s) {
    probe_kernel<<<1, 1024, SM_FLOATS * 4, s>>>(A, t, dt, out);
}

// The strip forms of the face pass: the same faces, a strip of H rows of a tile at a time (H = 16: halves, H = 8:
// quarters). A unit of work is one strip of a tile of the work list (32 / H units a tile); a CTA of 16 H threads (H / 2
// warps, two rows a warp) stages the strip with TMA as eight 40-column boxes of the rows each state field is read at
// (StripImage), its momenta as 32 x H boxes and its twelve static face scalars as bulk copies: 51 KB for 16 rows, so
// that four CTAs share a SM, 27 KB for 8 rows, eight (with 64 registers a thread). While one CTA waits for its copies
// the others compute (the tile form's two CTAs of 109 KB leave a SM idle whenever both wait). The plan shares, wanted
// on refresh steps only, are read from
// global memory. A face's arithmetic is the tile form's, bit for bit. On refresh steps each strip's wave maximum goes
// to its tile's entry and its run's maximum by integer atomic maxima on the float bits.
// Copy c of a strip's image, from the strip's first row y and its box's first column x0: the state boxes, the momenta (or
// the last step's mean depth box) and the twelve face scalars from table tile ts.
constexpr int STRIP_COPIES = 22;
template <int H>
__device__ __forceinline__ void strip_copy(int c, const StripMaps& M, const StepArgs& A, float* sm, uint64_t* bar, int x0,
                                           int y, int p, int mst, int ts, int row0) {
    using L = StripImage<H>;
    if (c < 12) {
        const int ax = c >= 6, f = c - 6 * ax;
        const float* from = f == 0 ? A.fl[ax] : f == 1 ? A.fr[ax] : f == 2 ? A.gl[ax] : f == 3 ? A.gr[ax]
                          : f == 4 ? A.ef[ax] : A.cw[ax];
        bulk_load(sm + L::ST + c * L::S, from + (size_t)ts * TILE2 + row0 * TILE, L::S * 4, bar);
        return;
    }
    switch (c) {
        case 12: tma_load_2d(sm + L::S_U, &M.u[p], x0, y - 2, bar); break;
        case 13: tma_load_2d(sm + L::S_V, &M.v[p], x0, y - 2, bar); break;
        case 14: tma_load_2d(sm + L::S_D, &M.d, x0, y - 1, bar); break;
        case 15: tma_load_2d(sm + L::S_H, &M.h[p], x0, y - 1, bar); break;
        case 16: tma_load_2d(sm + L::S_QX, &M.qx, x0, y - 1, bar); break;
        case 17: tma_load_2d(sm + L::S_QY, &M.qy, x0, y - 1, bar); break;
        case 18: tma_load_2d(sm + L::S_ZCX, &M.zcx, x0, y, bar); break;
        case 19: tma_load_2d(sm + L::S_ZCY, &M.zcy, x0, y - 1, bar); break;
        case 20:
            if (mst)
                tma_load_2d(sm + L::M, &M.mx[p], x0 + 4, y, bar);
            else
                tma_load_2d(sm + L::M, &M.h[1 - p], x0, y - 1, bar);  // the mean depth box's rows
            break;
        case 21:
            if (mst) tma_load_2d(sm + L::M + L::S, &M.my[p], x0 + 4, y, bar);
            break;
    }
}

// One strip of tile t at (tj, ti), with the tables of tile ts, from its row row0 on: its copies, then WARPS warps' rows of
// both faces, and on refresh steps the strip's wave maximum. SPREAD: each warp issues its share of the copies, and with
// more warps than rows a warp takes one axis of its row. False: the copies did not land (reported; the caller leaves).
template <int H, int WARPS, bool ON, bool SPREAD>
__device__ __forceinline__ bool strip_unit(const StripMaps& SM_, const StepArgs& A, float* sm, uint64_t* bar,
                                           uint32_t& phase, const float* rowc, float* red, int t, int ts, int tj, int ti,
                                           int row0, int run, float dt, float dx, int want_wave, int p, int mst,
                                           uint32_t* wave_bits) {
    using L = StripImage<H>;
    constexpr bool SPLIT = WARPS > H;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (SPREAD) {
        if (lane == 0) {
            fence_proxy_async();
            if (warp == 0) mbar_expect_tx(bar, (uint32_t)(mst ? L::BYTES : L::BYTES_HO));
            for (int c = warp; c < STRIP_COPIES; c += WARPS)
                strip_copy<H>(c, SM_, A, sm, bar, ti * TILE + GX - 4, tj * TILE + GY + row0, p, mst, ts, row0);
        }
    } else if (tid == 0) {
        const float* statics[12] = {A.fl[0], A.fr[0], A.gl[0], A.gr[0], A.ef[0], A.cw[0],
                                    A.fl[1], A.fr[1], A.gl[1], A.gr[1], A.ef[1], A.cw[1]};
        fence_proxy_async();
        mbar_expect_tx(bar, (uint32_t)(mst ? L::BYTES : L::BYTES_HO));
        // each box from its first row (the strip's row 0 is y)
        const int x0 = ti * TILE + GX - 4, y = tj * TILE + GY + row0;
        tma_load_2d(sm + L::S_U, &SM_.u[p], x0, y - 2, bar);
        tma_load_2d(sm + L::S_V, &SM_.v[p], x0, y - 2, bar);
        tma_load_2d(sm + L::S_D, &SM_.d, x0, y - 1, bar);
        tma_load_2d(sm + L::S_H, &SM_.h[p], x0, y - 1, bar);
        tma_load_2d(sm + L::S_QX, &SM_.qx, x0, y - 1, bar);
        tma_load_2d(sm + L::S_QY, &SM_.qy, x0, y - 1, bar);
        tma_load_2d(sm + L::S_ZCX, &SM_.zcx, x0, y, bar);
        tma_load_2d(sm + L::S_ZCY, &SM_.zcy, x0, y - 1, bar);
        if (mst) {
            tma_load_2d(sm + L::M, &SM_.mx[p], x0 + 4, y, bar);
            tma_load_2d(sm + L::M + L::S, &SM_.my[p], x0 + 4, y, bar);
        } else {
            tma_load_2d(sm + L::M, &SM_.h[1 - p], x0, y - 1, bar);  // the mean depth box's rows
        }
        for (int f = 0; f < 12; ++f)
            bulk_load(sm + L::ST + f * L::S, statics[f] + (size_t)ts * TILE2 + row0 * TILE, L::S * 4, bar);
    }
    const bool ok = mbar_wait(bar, phase);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
        // the copies did not land: report, and give them one more bounded wait before the CTA leaves
        if (tid == 0) atomicExch(&A.ctl->status, W2B_ETIMEOUT);
        mbar_wait(bar, phase ^ 1u);
        return false;
    }
    const int base = (tj * TILE + GY) * A.px + ti * TILE + GX;
    float wmax = 0.0f;
    if (SPLIT) {
        const int js = warp >> 1, ii = lane;
        const int jj = row0 + js;
        const int sl = js * TILE + ii, local = jj * TILE + ii;
        const int b = (js + 2) * BOXW + ii + 4;
        const int k = base + jj * A.px + ii;
        FaceA f;
        if (warp & 1) {
            face_a<1, ON, L>(sm, b, sl, local, A, ts, f);
            wmax = face_bc<1, false, ON, L>(sm, b, sl, local, k, A, ts, f, dt, dx, want_wave, rowc, p, mst);
        } else {
            face_a<0, ON, L>(sm, b, sl, local, A, ts, f);
            wmax = face_bc<0, false, ON, L>(sm, b, sl, local, k, A, ts, f, dt, dx, want_wave, rowc, p, mst);
        }
    }
#pragma unroll 1
    for (int c = 0; c < (SPLIT ? 0 : H / WARPS); ++c) {
        const int js = warp + WARPS * c, ii = lane;  // the row in the strip, and in the tile
        const int jj = row0 + js;
        const int sl = js * TILE + ii, local = jj * TILE + ii;
        const int b = (js + 2) * BOXW + ii + 4;
        const int k = base + jj * A.px + ii;
        FaceA fx, fy;
        face_a<0, ON, L>(sm, b, sl, local, A, ts, fx);
        face_a<1, ON, L>(sm, b, sl, local, A, ts, fy);
        const float wx = face_bc<0, false, ON, L>(sm, b, sl, local, k, A, ts, fx, dt, dx, want_wave, rowc, p, mst);
        const float wy = face_bc<1, false, ON, L>(sm, b, sl, local, k, A, ts, fy, dt, dx, want_wave, rowc, p, mst);
        wmax = fmax32(wmax, fmax32(wx, wy));
    }
    if (want_wave) {
        const float bm = block_max(wmax, red);
        if (tid == 0) {
            atomicMax(reinterpret_cast<unsigned int*>(A.wave) + t, __float_as_uint(bm));
            atomicMax(wave_bits + run, __float_as_uint(bm));
        }
    } else {
        __syncthreads();
    }
    return true;
}

// Where a CTA's next tiles or strips lie, with their runs' settings: a chain of dependent loads (work list -> tile -> its
// run -> its settings), each from L2. A CTA takes the chains of several at once into shared memory, a thread each, so that
// a unit's copies are issued as soon as the one before it is done: a step at 4096^2 takes 843 us against 860 with each
// unit's chain before its copies, at 1500 x 1101 125.2 against 126.2.
struct Place {
    int t, ts, run, tj, ti;
    int flags_p;  // the run's flags and its half (bit 31)
    float dt, dx;
};
__device__ __forceinline__ Place take_place(const StepArgs& A, int t) {
    Place W;
    W.t = t;
    W.run = A.tile_run[t];
    W.ts = table_of(A, t);
    W.tj = A.tiles[2 * t];
    W.ti = A.tiles[2 * t + 1];
    W.flags_p = A.R.flags[W.run] | (A.R.parity[W.run] << 31);
    W.dt = A.R.dtf[W.run];
    W.dx = A.R.dx[W.run];
    return W;
}
constexpr int STRIP_PLACES = 8;  // as many as leave eight CTAs of eight rows on a SM

template <int H, bool ON>
__global__ void __launch_bounds__(StripImage<H>::THREADS, StripImage<H>::CTAS)
    strips_kernel(const __grid_constant__ StripMaps M, StepArgs A) {
    using L = StripImage<H>;
    constexpr int PER = TILE / H;  // strips a tile
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ float red[L::THREADS / 32];
    __shared__ float rowc[2 * 64 + 1];
    __shared__ Place places[STRIP_PLACES];
    Ctl* ctl = A.ctl;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    fill_rowc(rowc, A.rows);
    __syncthreads();
    if (!(*A.any & ANY_RUN)) return;
    const int nunits = PER * ctl->nwork;
    const int mst = ctl->m_stored;
    uint32_t phase = 0;
    const int G = gridDim.x;
    for (int u0 = blockIdx.x; u0 < nunits; u0 += STRIP_PLACES * G) {
        if (threadIdx.x < STRIP_PLACES && u0 + (int)threadIdx.x * G < nunits)
            places[threadIdx.x] = take_place(A, A.list[(u0 + (int)threadIdx.x * G) / PER]);
        __syncthreads();
        for (int i = 0; i < STRIP_PLACES && u0 + i * G < nunits; ++i) {
            const Place& W = places[i];
            const int flags = W.flags_p & 0x7fffffff;
            if (!(flags & F_RUN)) continue;  // the tile's run has finished: uniform over the CTA
            if (!strip_unit<H, L::THREADS / 32, ON, false>(M, A, sm, &bar, phase, rowc, red, W.t, W.ts, W.tj, W.ti,
                                                           ((u0 + i * G) % PER) * H, W.run, W.dt, W.dx,
                                                           (flags & F_WAVE) != 0, W.flags_p < 0, mst, A.R.wave_bits))
                return;
        }
        __syncthreads();  // every thread has read the places
    }
}

cudaError_t faces_setup() {
    cudaError_t e = cudaFuncSetAttribute(probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_FLOATS * 4);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(faces_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    FACES_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(faces_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    FACES_SMEM);
    for (auto k : {strips_kernel<16, true>, strips_kernel<16, false>}) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, StripImage<16>::SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
    for (auto k : {strips_kernel<8, true>, strips_kernel<8, false>}) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, StripImage<8>::SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
    return e;
}

// The resident CTAs a SM of the strip form of `rows` rows (16 or 8).
int strips_occupancy(int rows) {
    int on = 0, off = 0;
    if (rows == 16) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&on, strips_kernel<16, true>, StripImage<16>::THREADS,
                                                      StripImage<16>::SMEM);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&off, strips_kernel<16, false>, StripImage<16>::THREADS,
                                                      StripImage<16>::SMEM);
    } else {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&on, strips_kernel<8, true>, StripImage<8>::THREADS,
                                                      StripImage<8>::SMEM);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&off, strips_kernel<8, false>, StripImage<8>::THREADS,
                                                      StripImage<8>::SMEM);
    }
    return on < off ? on : off;
}

// The face pass in its strip form of `rows` rows (16 or 8); grid: CTAs (the units are the work list's tiles, 32 /
// rows strips each).
void launch_strips(int rows, const TMaps& M, const StepArgs& A, int grid, cudaStream_t s) {
    const bool on = A.P.second && A.P.sheet && A.P.mirror && A.P.carry;
    if (rows == 16) {
        if (on)
            strips_kernel<16, true><<<grid, StripImage<16>::THREADS, StripImage<16>::SMEM, s>>>(M.s16, A);
        else
            strips_kernel<16, false><<<grid, StripImage<16>::THREADS, StripImage<16>::SMEM, s>>>(M.s16, A);
    } else {
        if (on)
            strips_kernel<8, true><<<grid, StripImage<8>::THREADS, StripImage<8>::SMEM, s>>>(M.s8, A);
        else
            strips_kernel<8, false><<<grid, StripImage<8>::THREADS, StripImage<8>::SMEM, s>>>(M.s8, A);
    }
}

// The resident CTAs a SM of the face pass (the smaller of its two forms').
int faces_occupancy() {
    int on = 0, off = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&on, faces_kernel<true>, FACES_THREADS, FACES_SMEM);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&off, faces_kernel<false>, FACES_THREADS, FACES_SMEM);
    return on < off ? on : off;
}

// The face pass, in its form with the numerics switches folded in when they are all on (the reference's defaults).
void launch_faces(const TMaps& M, const StepArgs& A, int grid, cudaStream_t s) {
    if (A.P.second && A.P.sheet && A.P.mirror && A.P.carry)
        faces_kernel<true><<<grid, FACES_THREADS, FACES_SMEM, s>>>(M.tile, A);
    else
        faces_kernel<false><<<grid, FACES_THREADS, FACES_SMEM, s>>>(M.tile, A);
}

// ------------------------------------------------------------------ update pass

__device__ __forceinline__ float scaled(float q, float rl, float rr) { return q * (q > 0.0f ? rl : rr); }

constexpr int RING = TILE + 2;  // the tile and its one-cell ring
constexpr int RPAD = RING + 1;
constexpr int U_QX1 = 0, U_QY1 = 1, U_H = 2;       // 40 x 36 boxes
constexpr int U_OWN = 3 * BOX;                      // res, src, hc: 32 x 32 each
constexpr int U_R = U_OWN + 3 * TILE2;              // r of the tile and its ring
constexpr int U_LP = (U_R + RING * RPAD + 31) / 32 * 32;  // the tile's cached level pairs (float2), 128-byte aligned
constexpr int U_LR = U_LP + 2 * TILE2;                     // and their rows (bytes)
constexpr int U_FLOATS = U_LR + TILE2 / 4;
constexpr int UPDATE_SMEM = U_FLOATS * 4;           // 43,648 bytes: four CTAs a SM
static_assert(UPDATE_SMEM == 43648, "update image size");
constexpr int UPDATE_THREADS = 256;

// The positivity ratio r (wadi2d/solver/gpu/kernels/cells.cu:4-19) of the cell at box index b, from the unscaled
// discharges and the old depth.
__device__ __forceinline__ float positivity(const float* QX1, const float* QY1, const float* H, int b, float dt,
                                            float area) {
    const float out = fmax32(QX1[b + 1], 0.0f) + fmax32(-QX1[b], 0.0f) + fmax32(QY1[b + BOXW], 0.0f) +
                      fmax32(-QY1[b], 0.0f);
    const float have = fmax32(H[b], 0.0f) * area;
    return out * dt > have ? have / (out * dt) : 1.0f;
}

// What continuity hands to the level lookup: the new mean depth, its table row (-1: none, Hc <= 0), the row coordinate.
struct CellOut {
    float hn, sv, hc;
    int row;
};

// Continuity (cells.cu:219-232) of the cell at box index b, own index `local` and native index k: the scaled discharges,
// the residual and the mean depth written, and the level table's row (common.cuh cell_level): the top row above Hc.
// row: r of the cell in the ring's image. prescribed: a boundary cell whose depths another thread writes.
__device__ __forceinline__ CellOut continuity(const StepArgs& A, const float* QX1, const float* QY1, const float* H,
                                              const float* row, int b, int local, int k, const float* RES,
                                              const float* SRC, const float* HC, float* h_next, float dt, float area,
                                              bool prescribed = false) {
    const int last = A.rows - 1;
    CellOut C;
    const float rc = row[0];
    const float qw = scaled(QX1[b], row[-1], rc);
    const float qe = scaled(QX1[b + 1], rc, row[1]);
    const float qn = scaled(QY1[b], row[-RPAD], rc);
    const float qs = scaled(QY1[b + BOXW], rc, row[RPAD]);
    A.q[0][k] = qw;
    A.q[1][k] = qn;
    const float h0 = H[b];
    const float inc = RES[local] + dt * SRC[local] - dt * (qe - qw + qs - qn) / area;
    const float total = h0 + inc;
    C.hn = fmax32(total, 0.0f);
    A.res[k] = total > 0.0f ? inc - (total - h0) : 0.0f;
    if (!prescribed) h_next[k] = C.hn;
    const float hcv = HC[local];
    C.hc = hcv;
    if (hcv <= 0.0f) {
        C.row = -1;
        C.sv = 0.0f;
    } else if (C.hn >= hcv) {
        C.row = last - 1;
        C.sv = -1.0f;
    } else {
        C.sv = sqrtf(C.hn / hcv) * (float)last;
        C.row = row_of(C.sv, last);
    }
    return C;
}

// The cell's level pair: the cached one where its row is the cached row (about 699 cells in 700 from one step to the
// next), else gathered from the table and cached. fid: the cell in the cache's arrays, local: in the tile's table.
__device__ __forceinline__ float2 level_pair(const StepArgs& A, const float2* pairs_t, const float2* LP,
                                             const uint8_t* LR, int own, int row, size_t fid, int local) {
    if (row < 0) return make_float2(0.0f, 0.0f);
    if (LR[own] == row) return LP[own];
    const float2 pr = __ldg(pairs_t + (size_t)row * TILE2 + local);
    A.lpair[fid] = pr;
    A.lrow[fid] = (uint8_t)row;
    return pr;
}

// The level of a cell, and its wet share into om.
__device__ __forceinline__ float cell_out_level(const StepArgs& A, const CellOut& C, float2 q, float& om) {
    const int last = A.rows - 1;
    float dk;
    om = 1.0f;
    if (C.hc <= 0.0f) {
        dk = C.hn;
    } else if (C.hn >= C.hc) {
        dk = q.y + (C.hn - C.hc);
    } else {
        const int r = C.row;
        if (A.P.level_fp64 && r == 0) {
            const double sd = sqrt((double)C.hn / (double)C.hc) * (double)last;
            dk = (float)((double)q.x + sd * ((double)q.y - (double)q.x));
        } else {
            dk = q.x + (C.sv - (float)r) * (q.y - q.x);
        }
        const float m = (float)last;
        om = C.hc * (float)(2 * r + 1) / (m * m) / fmax32(q.y - q.x, 1e-12f);
    }
    return dk;
}

// Issue (thread 0) the copies of a tile's update image against bar: the unscaled discharges and the old depth with
// their ring, the residual, the source and Hc, and the tile's level cache (each cell's last level pair and its row).
__device__ __forceinline__ void update_issue(float* sm, uint64_t* bar, const UpdateMaps& M, const StepArgs& A,
                                             const Place& W) {
    const int p = W.flags_p < 0, tj = W.tj, ti = W.ti, t = W.t;
    fence_proxy_async();
    mbar_expect_tx(bar, (uint32_t)(3 * BOX + 3 * TILE2) * 4u + (uint32_t)TILE2 * 9u);
    const int x0 = ti * TILE + GX - 4, y0 = tj * TILE + GY - 2;
    tma_load_2d(sm + U_QX1 * BOX, &M.qx1, x0, y0, bar);
    tma_load_2d(sm + U_QY1 * BOX, &M.qy1, x0, y0, bar);
    tma_load_2d(sm + U_H * BOX, &M.h[p], x0, y0, bar);
    tma_load_2d(sm + U_OWN, &M.res, x0 + 4, y0 + 2, bar);
    tma_load_2d(sm + U_OWN + TILE2, &M.src, x0 + 4, y0 + 2, bar);
    bulk_load(sm + U_OWN + 2 * TILE2, A.hc + (size_t)W.ts * TILE2, TILE2 * 4, bar);
    bulk_load(sm + U_LP, A.lpair + (size_t)t * TILE2, TILE2 * 8, bar);
    bulk_load(sm + U_LR, A.lrow + (size_t)t * TILE2, TILE2, bar);
}

// The update pass (wadi2d/solver/gpu/kernels/cells.cu:4-63 with limit fused in): TMA stages the tile's unscaled
// discharges and old depth with their ring, its residual, source and Hc, and its level cache; r of the tile and its
// one-cell ring is formed in shared memory; then each thread takes its four cells through continuity and takes their
// level pairs from the cache, or for the cells whose row changed from the table (the gathers issued together). Once
// every thread has read the image, thread 0 issues the next tile's copies into it, and they land while any gathers
// return and the level, the wet share and the wet flag are finished.
// Four CTAs a SM: 64 registers. Three (69) took half of the places' gain, five (48, with spills) 3 % of a step.
constexpr int UPDATE_PLACES = 16;
// control: a step of the device loop, whose first CTA takes no tiles but forms the next step's settings meanwhile (they
// need the face pass's wave maxima only). As a kernel of its own at the step's end that work, a chain of loads and FP64
// in one CTA, was 8-14 us of every step.
__global__ void __launch_bounds__(UPDATE_THREADS, 4) update_kernel(const __grid_constant__ UpdateMaps M, StepArgs A,
                                                                int control) {
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ Place places[2 * UPDATE_PLACES];
    Ctl* ctl = A.ctl;
    const int px = A.px;
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    grid_open();
    const int worker = (int)blockIdx.x - control, workers = (int)gridDim.x - control;
    if (worker < 0) {
        next_settings(A, step_view(A.R, 0), step_view(A.R, 1), *A.any, A.any_next, grid_state(ctl));
        return;
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (!(*A.any & ANY_RUN)) return;
    const int nwork = ctl->nwork;
    // the face pass before this one has stepped: from now on the momenta are formed from the state (Ctl::m_stored)
    if (worker == 0 && tid == 0) ctl->m_stored = 0;
    uint32_t phase = 0;
    const float* QX1 = sm + U_QX1 * BOX;
    const float* QY1 = sm + U_QY1 * BOX;
    const float* H = sm + U_H * BOX;
    const float* RES = sm + U_OWN;
    const float* SRC = sm + U_OWN + TILE2;
    const float* HC = sm + U_OWN + 2 * TILE2;
    float* rs = sm + U_R;
    const int n = worker < nwork ? (nwork - worker + workers - 1) / workers : 0;  // this CTA's tiles
    // the places of UPDATE_PLACES of them from `first` on, into their half of the ring
    auto take = [&](int first) {
        const int i = first + tid;
        if (tid < UPDATE_PLACES && i < n)
            places[i % (2 * UPDATE_PLACES)] = take_place(A, A.list[worker + i * workers]);
    };
    take(0);
    __syncthreads();
    if (tid == 0 && n > 0) update_issue(sm, &bar, M, A, places[0]);
    for (int i = 0; i < n; ++i) {
        if (i % UPDATE_PLACES == 0) take(i + UPDATE_PLACES);  // (their half was last read at tile i - 1)
        const Place& W = places[i % (2 * UPDATE_PLACES)];
        const int t = W.t, ts = W.ts, tj = W.tj, ti = W.ti, p = W.flags_p < 0;
        const int flags = W.flags_p & 0x7fffffff;
        const float dt = W.dt, dxr = W.dx;
        const float area = dxr * dxr;
        const int want_plan = (flags & F_WAVE) != 0;
        const int want_wet = (flags & F_WET) != 0;
        float* __restrict__ h_next = A.hh[1 - p];
        const bool ok = mbar_wait(&bar, phase);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicExch(&ctl->status, W2B_ETIMEOUT);
            mbar_wait(&bar, phase ^ 1u);
            return;
        }
        if (!(flags & F_RUN)) {  // the tile's run has finished: uniform over the CTA
            __syncthreads();
            if (tid == 0 && i + 1 < n) update_issue(sm, &bar, M, A, places[(i + 1) % (2 * UPDATE_PLACES)]);
            continue;
        }
        // r of the tile and its ring, from the old h
        for (int idx = tid; idx < RING * RING; idx += UPDATE_THREADS) {
            const int rj = idx / RING, ri = idx - rj * RING;
            rs[rj * RPAD + ri] = positivity(QX1, QY1, H, (rj + 1) * BOXW + ri + 3, dt, area);  // cell (rj - 1, ri - 1)
        }
        __syncthreads();
        const int base = (tj * TILE + GY) * px + ti * TILE + GX;
        const float2* __restrict__ pairs_t = A.dtab2 + (size_t)ts * (A.rows - 1) * TILE2;
        CellOut C[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int jj = ty * 4 + c, ii = tx;
            C[c] = continuity(A, QX1, QY1, H, rs + (jj + 1) * RPAD + (ii + 1), (jj + 2) * BOXW + ii + 4, jj * TILE + ii,
                              base + jj * px + ii, RES, SRC, HC, h_next, dt, area);
        }
        float2 pr[4];
        const float2* LP = reinterpret_cast<const float2*>(sm + U_LP);
        const uint8_t* LR = reinterpret_cast<const uint8_t*>(sm + U_LR);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int local = (ty * 4 + c) * TILE + tx;
            pr[c] = level_pair(A, pairs_t, LP, LR, local, C[c].row, (size_t)t * TILE2 + local, local);
        }
        // every thread has read the image and r: the next tile's copies land in it during this tile's gathers
        __syncthreads();
        if (tid == 0 && i + 1 < n) update_issue(sm, &bar, M, A, places[(i + 1) % (2 * UPDATE_PLACES)]);
        int any = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int k = base + (ty * 4 + c) * px + tx;
            float om;
            A.d[k] = cell_out_level(A, C[c], pr[c], om);
            if (want_plan) A.om[k] = om;
            any |= C[c].hn > 0.0f;
        }
        if (want_wet) {
            const int w = __syncthreads_or(any);
            if (tid == 0) A.wet[t] = w;
        }
    }
}

cudaError_t update_setup() {
    return cudaFuncSetAttribute(update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, UPDATE_SMEM);
}

int update_occupancy() {
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, update_kernel, UPDATE_THREADS, UPDATE_SMEM);
    return occ;
}

// grid: the CTAs, with control (a step of the device loop) at least two.
void launch_update(const TMaps& M, const StepArgs& A, int grid, int control, cudaStream_t s) {
    update_kernel<<<grid, UPDATE_THREADS, UPDATE_SMEM, s>>>(M.update, A, control);
}

// ------------------------------------------------------------------ the resident loop

// Shared-memory image of a strip of H rows for the resident loop's update: boxes of 40 x (H + 3) floats from one row
// above the strip to two below (own cell (j, i) at box (j + 1, i + 4)), the own rows' residual, source and Hc, r of the
// strip and its one-cell ring, and the level cache.
template <int H>
struct UpdateStrip {
    static constexpr int BOXN = pad32(BOXW * (H + 3));
    static constexpr int QX1 = 0, QY1 = BOXN, HB = 2 * BOXN, RES = 3 * BOXN, SRC = RES + TILE * H, HC = SRC + TILE * H;
    static constexpr int R = HC + TILE * H, LP = pad32(R + (H + 2) * RPAD), LR = LP + 2 * TILE * H;
    static constexpr int SMEM = 4 * LR + TILE * H;
    static constexpr int BYTES = 4 * (3 * BOXW * (H + 3) + 3 * TILE * H) + 9 * TILE * H;
    static constexpr int CELLS = H * TILE / RESIDENT_THREADS > 0 ? H * TILE / RESIDENT_THREADS : 1;  // a thread
};

// A unit of the resident loop, a strip of H rows of a tile: where it lies, and its run's settings.
struct Unit {
    int t, run, ts, tj, ti, row0;
};
struct UnitStep {
    float dt, dx;
    int flags, p;
};
constexpr int UNITS_HELD = 32;  // units whose places a CTA keeps from step to step

template <int H>
__device__ __forceinline__ Unit unit_place(const StepArgs& A, int u) {
    constexpr int PER = TILE / H;
    Unit U;
    U.t = __ldcg(A.work + u / PER);
    U.run = A.tile_run[U.t];
    U.ts = table_of(A, U.t);
    U.tj = A.tiles[2 * U.t];
    U.ti = A.tiles[2 * U.t + 1];
    U.row0 = (u % PER) * H;
    return U;
}

__device__ __forceinline__ UnitStep unit_step(const StepArgs& A, const StepView& V, int run) {
    return UnitStep{__ldcg(V.dtf + run), A.R.dx[run], __ldcg(V.flags + run), __ldcg(V.parity + run)};
}

// The update of one strip with its envelope; the update pass's arithmetic. leave: the depths of a boundary cell (bmark) are
// left to whoever takes it (boundary_items), so that neither waits for the other. What does not depend on the copies (the
// marks, the envelope's entries, and `meanwhile`) is done while they land. False: they did not land (reported; the caller
// leaves).
template <int H, class Meanwhile>
__device__ __forceinline__ bool update_unit(const UpdateMaps& M, const StepArgs& A, const StepView& V, float* sm,
                                            uint64_t* bar, uint32_t& phase, const Unit& U, const UnitStep& S, bool leave,
                                            Meanwhile meanwhile) {
    using L = UpdateStrip<H>;
    const int tid = threadIdx.x, px = A.px;
    const float dt = S.dt, area = S.dx * S.dx;
    const int want_max = (S.flags & F_MAX) == F_MAX, n = 1 - S.p;
    const int base = (U.tj * TILE + GY + U.row0) * px + U.ti * TILE + GX;  // the strip's first cell
    const size_t fid0 = (size_t)U.t * TILE2 + U.row0 * TILE;
    if ((tid & 31) == 0) {
        const int x0 = U.ti * TILE + GX - 4, y0 = U.tj * TILE + GY + U.row0;
        fence_proxy_async();
        switch (tid >> 5) {
            case 0:
                mbar_expect_tx(bar, (uint32_t)L::BYTES);
                tma_load_2d(sm + L::QX1, &M.qx1, x0, y0 - 1, bar);
                break;
            case 1: tma_load_2d(sm + L::QY1, &M.qy1, x0, y0 - 1, bar); break;
            case 2: tma_load_2d(sm + L::HB, &M.h[S.p], x0, y0 - 1, bar); break;
            case 3: tma_load_2d(sm + L::RES, &M.res, x0 + 4, y0, bar); break;
            case 4: tma_load_2d(sm + L::SRC, &M.src, x0 + 4, y0, bar); break;
            case 5:
                bulk_load(sm + L::HC, A.hc + (size_t)U.ts * TILE2 + U.row0 * TILE, TILE * H * 4, bar);
                break;
            case 6: bulk_load(sm + L::LP, A.lpair + fid0, TILE * H * 8, bar); break;
            case 7: bulk_load(sm + L::LR, A.lrow + fid0, TILE * H, bar); break;
        }
    }
    const bool mine = tid < H * TILE;
    EnvelopeIn E[L::CELLS];
    uint32_t marked[L::CELLS];
#pragma unroll
    for (int c = 0; c < L::CELLS; ++c) {
        const int cell = tid + RESIDENT_THREADS * c, js = cell >> 5, ii = cell & 31;
        marked[c] = mine && A.nb ? (A.bmark[U.t * TILE + U.row0 + js] >> ii) & 1u : 0u;
        if (mine && want_max) E[c] = envelope_load(A, (int)fid0 + cell, base + js * px + ii, A.uu[0][n], A.uu[1][n]);
    }
    float time = 0.0f, arrive = 0.0f, deep = 0.0f;
    if (want_max) time = __ldcg(V.max_time + U.run), arrive = A.ctl->arrive, deep = A.ctl->deep;
    meanwhile();
    const bool ok = mbar_wait(bar, phase);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) {
        if (tid == 0) atomicExch(&A.ctl->status, W2B_ETIMEOUT);
        mbar_wait(bar, phase ^ 1u);
        return false;
    }
    const float *QX1 = sm + L::QX1, *QY1 = sm + L::QY1, *HB = sm + L::HB;
    float* rs = sm + L::R;
    for (int idx = tid; idx < (H + 2) * RING; idx += RESIDENT_THREADS) {
        const int rj = idx / RING, ri = idx - rj * RING;
        rs[rj * RPAD + ri] = positivity(QX1, QY1, HB, rj * BOXW + ri + 3, dt, area);  // cell (rj - 1, ri - 1)
    }
    __syncthreads();
    const float2* pairs_t = A.dtab2 + (size_t)U.ts * (A.rows - 1) * TILE2 + U.row0 * TILE;
    const float2* LP = reinterpret_cast<const float2*>(sm + L::LP);
    const uint8_t* LR = reinterpret_cast<const uint8_t*>(sm + L::LR);
    int any = 0;
    if (mine) {
        CellOut C[L::CELLS];
        float2 pr[L::CELLS];
#pragma unroll
        for (int c = 0; c < L::CELLS; ++c) {
            const int cell = tid + RESIDENT_THREADS * c, js = cell >> 5, ii = cell & 31;
            C[c] = continuity(A, QX1, QY1, HB, rs + (js + 1) * RPAD + (ii + 1), (js + 1) * BOXW + ii + 4, cell,
                              base + js * px + ii, sm + L::RES, sm + L::SRC, sm + L::HC, A.hh[n], dt, area,
                              leave && marked[c]);
            pr[c] = level_pair(A, pairs_t, LP, LR, cell, C[c].row, fid0 + cell, cell);
        }
#pragma unroll
        for (int c = 0; c < L::CELLS; ++c) {
            const int cell = tid + RESIDENT_THREADS * c, k = base + (cell >> 5) * px + (cell & 31);
            float om;
            const float dk = cell_out_level(A, C[c], pr[c], om);
            if (!(leave && marked[c])) A.d[k] = dk;
            if (S.flags & F_WAVE) A.om[k] = om;
            any |= C[c].hn > 0.0f;
            if (want_max && !marked[c])
                envelope_apply(A, (int)fid0 + cell, E[c], dk, C[c].hn, time, arrive, deep);
        }
    }
    // the strip's cells are written and its image is read; whether any is wet
    const int w = __syncthreads_or(any);
    if ((S.flags & F_WET) && w && tid == 0) atomicOr(A.wet + U.t, 1);
    return true;
}

// Up to max_steps steps of the device loop in one cooperative launch. A step of the loop's kernels of their own is five
// dependent launches, which on a few hundred tiles cost more than their work; here it is two grid barriers: the face
// pass by strips of H rows (first barrier), then the update of the same strips with their envelope, the boundary cells
// shared out over the CTAs, while one CTA of its own forms the next step's settings in the second set (second barrier);
// that CTA then takes the tally and the lines while the next face pass runs. Where some boundary cell follows another, all
// of them (one more barrier), and steps that rebuild the lists (two or three more, one step in active_every) come after it.
// The same arithmetic in the same order for every cell, face and sum as the kernels of their own. What CTAs hand one
// another between barriers is read past L1 or by bulk copies. Latency bounds it on small grids (issue active 11 % at 62 x
// 62, 27 % at 256 x 256, a warp's time mostly at barriers), so strips of 4 rows (a warp a row and axis) serve the
// smallest, and a CTA keeps the places of its strips from step to step. A step of the exact build, this way and as
// kernels of their own: 4 tiles 11.2 against 20.3 us, 64 tiles 16.6 against 21.1, 121 tiles 19.7 against 22.6. Where the
// passes' own work fills the chip it loses (1,645 tiles: 149 against 109 us), and the launch tuner leaves it out.
// A host-driven step (host.flags not 0) is one step of it: the settings come with the launch, the tiles are the active
// list (in A.work's place, host.tiles of them), nothing but the swap of run 0's halves follows.
template <int H, bool ON>
__global__ void __launch_bounds__(RESIDENT_THREADS, resident_ctas(H))
    resident_kernel(const __grid_constant__ ResidentMaps M, const __grid_constant__ StepArgs A, int max_steps,
                    HostStep host) {
    constexpr int PER = TILE / H;
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ float red[RESIDENT_THREADS / 32];
    __shared__ float rowc[2 * 64 + 1];
    __shared__ Unit places[UNITS_HELD];
    __shared__ UnitStep steps[UNITS_HELD];
    Ctl* ctl = A.ctl;
    GridState* grid = grid_state(ctl);
    const int workers = (int)gridDim.x - 1;  // the last CTA forms the next step's settings and rebuilds the lists
    const bool control = (int)blockIdx.x == workers;
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    fill_rowc(rowc, A.rows);
    uint32_t phase = 0, met = 0;
    uint32_t any = host.flags ? ANY_RUN : ctl->any;
    int nwork = host.flags ? host.tiles : ctl->nwork, mst = ctl->m_stored, b = 0;
    bool moved = true;  // the work list is not the one `places` was taken from
    const bool follow = A.nb && *follow_flag(ctl);
    if (ctl->status) return;  // a wait before this launch gave up: the barrier's counters may be anything
    for (int step = 0; step < max_steps && (any & ANY_RUN); ++step) {
        const StepView V = step_view(A.R, b);
        const int left = PER * nwork - (int)blockIdx.x;
        const int units = control || left <= 0 ? 0 : (left + workers - 1) / workers;  // this CTA's
        // the places and settings of its units from c0 on (kept from the step before where they are all held and the
        // lists have not moved; the settings then came with the step's flags)
        auto take = [&](int c0) {
            const int n = units - c0 < UNITS_HELD ? units - c0 : UNITS_HELD;
            __syncthreads();
            if (tid < n && (moved || units > UNITS_HELD)) {
                places[tid] = unit_place<H>(A, (int)blockIdx.x + (c0 + tid) * workers);
                steps[tid] = host.flags ? UnitStep{host.dt, A.R.dx[0], host.flags, __ldcg(A.R.parity)}
                                        : unit_step(A, V, places[tid].run);
            }
            __syncthreads();
            return n;
        };
        for (int c0 = 0; c0 < units; c0 += UNITS_HELD) {
            const int n = take(c0);
            for (int i = 0; i < n; ++i) {
                const Unit U = places[i];
                const UnitStep S = steps[i];
                if (!(S.flags & F_RUN)) continue;  // uniform over the CTA
                if ((S.flags & F_WET) && U.row0 == 0 && tid == 0) A.wet[U.t] = 0;  // its strips' updates join their flags
                if (!strip_unit<H, RESIDENT_THREADS / 32, ON, true>(M.s, A, sm, &bar, phase, rowc, red, U.t, U.ts, U.tj,
                                                                    U.ti, U.row0, U.run, S.dt, S.dx,
                                                                    (S.flags & F_WAVE) != 0, S.p, mst, V.wave_bits))
                    return;
            }
        }
        moved = false;
        if (!grid_barrier(grid, ctl, met)) return;
        if (control && host.flags) {
            if (tid == 0) ctl->m_stored = 0;
        } else if (control) {
            next_settings(A, V, step_view(A.R, b ^ 1), any, &ctl->any, grid);
        }
        // this CTA's boundary cells, before or during its first strip: 32 a CTA (they lie apart in memory, and one SM takes
        // in few such lines at once), the first ones in the last CTAs, which are those without a strip where there are any
        bool bounds = !control && A.nb && !follow;
        auto bound = [&] {
            if (bounds)
                boundary_items(A, V, ((tid >> 5) * workers + workers - 1 - (int)blockIdx.x) * 32 + (tid & 31),
                               workers * RESIDENT_THREADS, host.flags);
            bounds = false;
        };
        if (!units) bound();
        for (int c0 = 0; c0 < units; c0 += UNITS_HELD) {
            const int n = units > UNITS_HELD ? take(c0) : units;
            for (int i = 0; i < n; ++i)
                if (!(steps[i].flags & F_RUN))
                    bound();
                else if (!update_unit<H>(M.u, A, V, sm, &bar, phase, places[i], steps[i], !follow, bound))
                    return;
        }
        if (!grid_barrier(grid, ctl, met)) return;
        if (host.flags) {
            if (follow) {
                boundary_items(A, V, (int)(blockIdx.x * RESIDENT_THREADS) + tid, (int)(gridDim.x * RESIDENT_THREADS),
                               host.flags);
                if (!grid_barrier(grid, ctl, met)) return;
            }
            if (control && tid == 0) A.R.parity[0] ^= 1;
            break;
        }
        const uint32_t next = __ldcg(&ctl->any);
        const int rebuild = __ldcg(&grid->rebuild);
        if (tid < units && units <= UNITS_HELD) steps[tid] = unit_step(A, step_view(A.R, b ^ 1), places[tid].run);
        if (follow) {
            boundary_items(A, V, (int)(blockIdx.x * RESIDENT_THREADS) + tid, (int)(gridDim.x * RESIDENT_THREADS));
            if (!grid_barrier(grid, ctl, met)) return;
        }
        if (control) tally_items(A, V, tid, RESIDENT_THREADS);
        if (rebuild) {
            if (!grid_barrier(grid, ctl, met)) return;
            if (control) rebuild_lists(A, V, false, (any & ANY_ACT) != 0, true);
            if (!grid_barrier(grid, ctl, met)) return;
            nwork = __ldcg(&ctl->nwork);
            const int woken = __ldcg(&ctl->nwoken);
            if (woken) {
                if (!control) plan_tiles(A, step_view(A.R, b ^ 1).parity, A.woken, woken, blockIdx.x, workers);
                if (!grid_barrier(grid, ctl, met)) return;
            }
            moved = true;
        }
        b ^= 1;
        mst = 0;
        any = next;
    }
    // the settings of the step that comes next where the other forms of the loop read them
    if (b) {
        if (!grid_barrier(grid, ctl, met)) return;
        if (control) adopt_settings(A);
    }
    grid_leave(grid);
}

template <int H>
constexpr int resident_smem() {
    return StripImage<H>::SMEM > UpdateStrip<H>::SMEM ? StripImage<H>::SMEM : UpdateStrip<H>::SMEM;
}

struct ResidentForm {
    const void* kernel;
    int smem;
};
static ResidentForm resident_form(int rows, bool on) {
    switch (rows) {
        case 16:
            return {on ? (const void*)resident_kernel<16, true> : (const void*)resident_kernel<16, false>,
                    resident_smem<16>()};
        case 8:
            return {on ? (const void*)resident_kernel<8, true> : (const void*)resident_kernel<8, false>,
                    resident_smem<8>()};
        default:
            return {on ? (const void*)resident_kernel<4, true> : (const void*)resident_kernel<4, false>,
                    resident_smem<4>()};
    }
}

cudaError_t resident_setup() {
    cudaError_t e = cudaSuccess;
    for (const int rows : {16, 8, 4})
        for (const bool on : {true, false}) {
            const ResidentForm f = resident_form(rows, on);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f.smem);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        }
    return e;
}

// The resident CTAs a SM of the resident loop with strips of `rows` rows (16, 8 or 4).
int resident_occupancy(int rows) {
    int least = 1 << 20;
    for (const bool on : {true, false}) {
        const ResidentForm f = resident_form(rows, on);
        int occ = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f.kernel, RESIDENT_THREADS, f.smem);
        least = occ < least ? occ : least;
    }
    return least;
}

// Up to max_steps steps in one cooperative launch of `grid` CTAs (at least two, at most as many as are resident at
// once, `occupancy` a SM); the control block's grid state starts at zero.
cudaError_t launch_resident(int rows, const ResidentMaps& M, const StepArgs& A, int grid, int occupancy, int max_steps,
                            const HostStep& host, cudaStream_t s) {
    const ResidentForm f = resident_form(rows, A.P.second && A.P.sheet && A.P.mirror && A.P.carry);
    ResidentMaps maps = M;
    StepArgs args = A;
    HostStep step = host;
    void* params[] = {&maps, &args, &max_steps, &step};
    return launch_in_turn(f.kernel, grid, RESIDENT_THREADS, params, f.smem, occupancy, s);
}

}  // namespace W2B_ARITH

#ifndef W2B_FAST
// ------------------------------------------------------------------ self-checks

// Every positive float from first (as bits) on: cbrt32 against the double path; out[0] counts mismatches,
// out[1..4] keep some mismatching inputs.
__global__ void cbrt_check_kernel(uint32_t first, uint32_t count, unsigned long long* out) {
    for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < count; n += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t bits = first + (uint32_t)n;
        const float x = __uint_as_float(bits);
        const float a = cbrt32(x);
        const float b = (float)cbrt((double)x);
        if (__float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b))) {
            const unsigned long long k = atomicAdd(out, 1ull);
            if (k < 4) out[1 + k] = bits;
        }
    }
}

void launch_cbrt_check(uint32_t first, uint32_t count, unsigned long long* out, cudaStream_t s) {
    cbrt_check_kernel<<<148 * 16, 256, 0, s>>>(first, count, out);
}

// The bounded wait's give-up path, run on purpose: thread 0 arms a barrier for 16 bytes that no copy will bring, so
// its phase cannot complete, and waits on it with mbar_wait for `polls` polls. Nothing is in flight, so the CTA may
// leave. out[0] = W2B_ETIMEOUT if the wait gave up (W2B_OK if it completed, which it cannot), out[1] = the clock
// cycles the wait took.
__global__ void wait_check_kernel(uint32_t polls, long long* out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    fence_barrier_init();
    mbar_expect_tx(&bar, 16);  // the one arrival, with 16 bytes still expected
    const long long t0 = clock64();
    const bool ok = mbar_wait(&bar, 0, polls);
    out[1] = clock64() - t0;
    out[0] = ok ? W2B_OK : W2B_ETIMEOUT;
}

void launch_wait_check(uint32_t polls, long long* out, cudaStream_t s) { wait_check_kernel<<<1, 32, 0, s>>>(polls, out); }

// ------------------------------------------------------------------ face momenta

// The face momenta into their arrays (each run's current half), as the face pass forms them once a face pass has
// stepped: the last step's abar * u, abar from the other half of the mean depth pair (the depths that step started
// from), rounded once. Every own face of every tile; nothing when the arrays already hold the momenta
// (Ctl::m_stored), so it may run before any read or write of the state; the last CTA to leave records that they do.
// HBM bounds it: a CTA a tile, a thread four cells in a row by 16-byte loads, 56 us for 16.8 M cells (20 B a cell, 6.0
// TB/s), where a thread a cell with the tile's place looked up for each took 145.
__global__ void __launch_bounds__(256) momentum_kernel(StepArgs A) {
    if (A.ctl->m_stored) return;
    const int jj = threadIdx.x >> 3, ii = (threadIdx.x & 7) * 4;
    for (int t = 1 + blockIdx.x; t < A.ntiles; t += gridDim.x) {  // tile 0 is the void tile
        const int run = A.tile_run[t];
        const size_t k = (size_t)(A.tiles[2 * t] * TILE + GY + jj) * A.px + A.tiles[2 * t + 1] * TILE + GX + ii;
        const int p = A.R.parity[run];
        const float dx = A.R.dx[run];
        const float* ho = A.hh[1 - p];
        auto four = [](const float* q) { return *reinterpret_cast<const float4*>(q); };
        const float4 h = four(ho + k), s = four(ho + k - A.px), u = four(A.uu[0][p] + k), v = four(A.uu[1][p] + k);
        const float w = ho[k - 1];
        auto mom = [&](float a, float b, float c) { return __fmul_rn(0.5f * (a + b) * dx, c); };
        *reinterpret_cast<float4*>(A.mm[0][p] + k) =
            make_float4(mom(w, h.x, u.x), mom(h.x, h.y, u.y), mom(h.y, h.z, u.z), mom(h.z, h.w, u.w));
        *reinterpret_cast<float4*>(A.mm[1][p] + k) =
            make_float4(mom(s.x, h.x, v.x), mom(s.y, h.y, v.y), mom(s.z, h.z, v.z), mom(s.w, h.w, v.w));
    }
    __syncthreads();
    GridState* grid = grid_state(A.ctl);
    if (threadIdx.x == 0 && atomicAdd(&grid->done, 1u) == gridDim.x - 1) {
        A.ctl->m_stored = 1;
        grid->done = 0;
    }
}

// The other halves of the sleeping tiles from their current ones, after a caller has had the state arrays in hand: the
// passes never write a sleeping tile, so what it holds has to be the same in both halves of its pairs (as it is where a
// tile has fallen asleep by itself: dry and still), or the step after next would find in it what a write to the current
// half meant to replace. A CTA a tile, a thread four cells in a row; written only where they differ. 4 us a call for 430 k
// sleeping cells.
__global__ void __launch_bounds__(256) asleep_kernel(StepArgs A) {
    const int jj = threadIdx.x >> 3, ii = (threadIdx.x & 7) * 4;
    for (int t = 1 + blockIdx.x; t < A.ntiles; t += gridDim.x) {
        if (A.is_act[t]) continue;
        const size_t k = (size_t)(A.tiles[2 * t] * TILE + GY + jj) * A.px + A.tiles[2 * t + 1] * TILE + GX + ii;
        const int p = A.R.parity[A.tile_run[t]];
        float* const pairs[3][2] = {{A.hh[p], A.hh[1 - p]}, {A.uu[0][p], A.uu[0][1 - p]}, {A.uu[1][p], A.uu[1][1 - p]}};
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const uint4 x = *reinterpret_cast<const uint4*>(pairs[f][0] + k);
            const uint4 y = *reinterpret_cast<const uint4*>(pairs[f][1] + k);
            if ((x.x ^ y.x) | (x.y ^ y.y) | (x.z ^ y.z) | (x.w ^ y.w))
                *reinterpret_cast<uint4*>(pairs[f][1] + k) = x;
        }
    }
}

void launch_asleep(const StepArgs& A, int sms, cudaStream_t s) { asleep_kernel<<<sms * 8, 256, 0, s>>>(A); }

void launch_momentum(const StepArgs& A, int sms, cudaStream_t s) {
    momentum_kernel<<<sms * 8, 256, 0, s>>>(A);
}

// ------------------------------------------------------------------ the end of a step

// After the update of a step of the device loop: the boundary cells of every running run with their envelope entries, the
// FP64 tally and the design lines, and, at a step that records it (F_MAX), the envelope of the own cells of the work
// list's tiles. Each item is independent of the others (a follow boundary reads an interior cell), so one kernel takes
// them all: the first as a grid-stride loop, then a CTA a tile at a time, a thread a cell.
// A tile's place (work list -> tile -> its run, its first own cell, its rows' boundary marks) is a chain of dependent
// loads, each from L2; the CTA stages it for ENV_CHUNK of its tiles at once in shared memory (all chains in flight
// together), so that a tile's own work waits on its run's flags (L1-resident) and then on its cells' data only.
constexpr int ENV_CHUNK = 64;
__global__ void __launch_bounds__(TILE2, 2) step_end_kernel(StepArgs A) {
    __shared__ int3 place[ENV_CHUNK];            // tile, run, native index of the tile's first own cell
    __shared__ uint32_t marks[ENV_CHUNK * TILE];  // the tile's boundary marks, a word a row
    Ctl* ctl = A.ctl;
    grid_open();
    grid_wait();
    const uint32_t any = *A.any;
    if (any & ANY_RUN) {
        const StepView V = step_view(A.R, 0);
        const int gtid = blockIdx.x * TILE2 + threadIdx.x, gstride = gridDim.x * TILE2;
        boundary_items(A, V, gtid, gstride);
        // (from the other end, so that few threads have both a boundary cell and a tally face)
        tally_items(A, V, (gridDim.x - 1 - blockIdx.x) * TILE2 + threadIdx.x, gstride);
    }
    if (!(any & ANY_MAX)) return;
    const int nwork = ctl->nwork;
    const float arrive = ctl->arrive, deep = ctl->deep;
    const int tid = threadIdx.x, jj = tid >> 5, ii = tid & 31;
    const int G = gridDim.x;
    const int mine = (nwork - (int)blockIdx.x + G - 1) / G;  // this CTA's tiles: work positions blockIdx.x + i G
    for (int c0 = 0; c0 < mine; c0 += ENV_CHUNK) {
        const int nc = min(ENV_CHUNK, mine - c0);
        if (tid < nc) {
            const int t = A.list[blockIdx.x + (c0 + tid) * G];
            place[tid] = make_int3(t, A.tile_run[t],
                                   (A.tiles[2 * t] * TILE + GY) * A.px + A.tiles[2 * t + 1] * TILE + GX);
        }
        __syncthreads();
        for (int q = tid; q < nc * TILE; q += TILE2) marks[q] = A.bmark[place[q / TILE].x * TILE + q % TILE];
        __syncthreads();
        for (int i = 0; i < nc; ++i) {
            const int3 w = place[i];
            const int run = w.y;
            if ((A.R.flags[run] & (F_RUN | F_MAX)) != (F_RUN | F_MAX)) continue;
            if ((marks[i * TILE + jj] >> ii) & 1u) continue;
            const int p = A.R.parity[run];
            const int k = w.z + jj * A.px + ii;
            envelope_cell(A, w.x * TILE2 + tid, k, A.d[k], A.hh[1 - p][k], A.R.max_time[run], arrive, deep,
                          A.uu[0][1 - p], A.uu[1][1 - p]);
        }
        __syncthreads();  // the chunk's places and marks are read by every thread before the next chunk's overwrite
    }
}

// The boundary cells after a host-driven step, and the swap of run 0's ping-pong pairs at its end
// (wadi2d/solver/gpu/backend.py:185-188), by the last CTA to leave.
__global__ void boundary_kernel(StepArgs A) {
    grid_open();
    grid_wait();
    if (!(*A.any & ANY_RUN)) return;
    boundary_items(A, step_view(A.R, 0), blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    __syncthreads();
    GridState* grid = grid_state(A.ctl);
    if (threadIdx.x == 0 && atomicAdd(&grid->done, 1u) == gridDim.x - 1) {
        A.R.parity[0] ^= 1;
        grid->done = 0;
    }
}

// ------------------------------------------------------------------ settings and lists (one CTA)

// Before a step of the device loop, for each run: the loop test and the step's settings
// (wadi2d/solver/stepper.py:106-111). The threads of one CTA; ctl->any gathers the runs' flags.
__device__ void step_settings(const StepArgs& A) {
    Ctl* ctl = A.ctl;
    __shared__ uint32_t any;
    if (threadIdx.x == 0) any = 0u;
    __syncthreads();
    const StepView V = step_view(A.R, 0);
    uint32_t mine = 0u;
    for (int r = threadIdx.x; r < A.nruns; r += blockDim.x) mine |= run_settings(A, V, r);
    if (mine) atomicOr(&any, mine);
    __syncthreads();
    if (threadIdx.x == 0) ctl->any = any;
    if (any & ANY_WAVE) clear_waves(A, V);
}

// A host-driven step of run 0 (the reference backend's step(dt, want_wave, want_wet)), with the tiles' waves cleared when
// it wants them. One CTA.
__global__ void __launch_bounds__(1024) setstep_kernel(StepArgs A, float dtf, int want_wave, int want_wet, int nact) {
    Ctl* ctl = A.ctl;
    if (threadIdx.x == 0) {
        ctl->nact = nact;
        ctl->nwork = nact;
        ctl->any = ANY_RUN | (want_wave ? ANY_WAVE : 0u);
        A.R.dtf[0] = dtf;
        A.R.flags[0] = F_RUN | (want_wave ? F_WAVE : 0) | (want_wet ? F_WET : 0);
        if (want_wave) A.R.wave_bits[0] = 0u;
    }
    if (want_wave)
        for (int t = threadIdx.x; t < A.ntiles; t += blockDim.x) A.wave[t] = 0.0f;
}

// Before the first step of the device loop, in one CTA of 1024 threads: the loop's settings (c; the stored-momenta flag
// stays), each run's clock (clocks and t_ends, or a single run's by value), the work list of the runs that take a step,
// and the first step's settings.
__global__ void __launch_bounds__(1024) begin_kernel(const __grid_constant__ StepArgs A, Ctl c, W2BClock one, double t_end,
                                                     long long max_steps, const W2BClock* clocks,
                                                     const double* t_ends) {
    const RunTab& R = A.R;
    if (threadIdx.x == 0) {
        c.m_stored = A.ctl->m_stored;
        *A.ctl = c;
        GridState* grid = grid_state(A.ctl);  // whatever a wait that gave up has left
        grid->arrived = grid->left = 0;
        grid->rebuild = 0;
    }
    for (int r = threadIdx.x; r < A.nruns; r += blockDim.x) {
        const W2BClock k = clocks ? clocks[r] : one;
        R.t[r] = k.t;
        R.dt[r] = k.dt;
        R.t_end[r] = t_ends ? t_ends[r] : t_end;
        R.nsteps[r] = k.nsteps;
        R.steps_run[r] = 0;
        R.max_steps[r] = max_steps;
        R.refresh_due[r] = k.refresh_due;
        R.status[r] = 0;
    }
    __syncthreads();
    rebuild_lists(A, step_view(A.R, 0), true, false, false);
    __syncthreads();
    step_settings(A);
}

// The end of a step of the device loop, in one CTA of 1024 threads: at a step that checks (or after which some run has
// stopped) the active-list rebuild with the woken tiles and the work list, which plan_kernel takes after it; and with
// adopt (the last of a launch of an odd number of steps) the next step's settings where the first step of a launch reads
// them.
__global__ void __launch_bounds__(1024) rebuild_kernel(const __grid_constant__ StepArgs A, int adopt) {
    grid_open();
    grid_wait();
    if (grid_state(A.ctl)->rebuild) rebuild_lists(A, step_view(A.R, 0), false, (*A.any & ANY_ACT) != 0, true);
    if (adopt) {
        __syncthreads();
        adopt_settings(A);
        if (threadIdx.x == 0) *A.any = *A.any_next;
    }
}

// refresh_plan of the listed tiles (wadi2d/solver/gpu/kernels/cells.cu:66-78) from the current mean depth. count < 0:
// the tiles that a rebuild at the end of this step of the device loop woke, by the next step's halves.
__global__ void __launch_bounds__(256) plan_kernel(StepArgs A, const int32_t* list, int count) {
    grid_open();
    grid_wait();
    const bool loop = count < 0;
    if (loop) count = grid_state(A.ctl)->rebuild ? A.ctl->nwoken : 0;
    plan_tiles(A, loop ? A.R.parity2 : A.R.parity, list, count, blockIdx.x, gridDim.x);
}

// Maxima.update over the active tiles, host-driven (wadi2d/engine/maxima.py:118-130): the current halves are the
// state after the step.
__global__ void __launch_bounds__(256) maxima_kernel(StepArgs A, float time, float arrive, float deep, int nact) {
    for (int a = blockIdx.x; a < nact; a += gridDim.x) {
        const int t = A.active[a];
        const int tj = A.tiles[2 * t], ti = A.tiles[2 * t + 1];
        const int base = (tj * TILE + GY) * A.px + ti * TILE + GX;
        for (int c = 0; c < 4; ++c) {
            const int jj = threadIdx.y * 4 + c, ii = threadIdx.x;
            const int k = base + jj * A.px + ii;
            const int pc = A.R.parity[A.tile_run[t]];
            envelope_cell(A, t * TILE2 + jj * TILE + ii, k, A.d[k], A.hh[pc][k], time, arrive, deep, A.uu[0][pc], A.uu[1][pc]);
        }
    }
}

// Tally.add, host-driven (wadi2d/engine/maxima.py:53-62).
__global__ void tally_kernel(StepArgs A, double dt) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= A.ntally) return;
    const float qv = A.taxis[m] ? A.q[1][A.tface[m]] : A.q[0][A.tface[m]];
    A.ttotal[m] += dt * (double)(A.tsign[m] * qv);
}

// ------------------------------------------------------------------ layout converters

// REF_TILE -> NATIVE, own cells of every allocated tile (halo entries of the reference layout are copies).
__global__ void ref_to_native_kernel(const float* __restrict__ ref, float* __restrict__ nat,
                                     const int32_t* __restrict__ tiles, int ntiles, int px) {
    const int t = blockIdx.x + 1;
    if (t >= ntiles) return;
    const int tj = tiles[2 * t], ti = tiles[2 * t + 1];
    for (int idx = threadIdx.x; idx < TILE2; idx += blockDim.x) {
        const int jj = idx / TILE, ii = idx % TILE;
        nat[(size_t)(tj * TILE + jj + GY) * px + ti * TILE + ii + GX] = ref[(size_t)t * 1296 + (jj + 2) * 36 + ii + 2];
    }
}

// NATIVE -> REF_TILE, every entry of every allocated tile: halos read the neighbour cell they copy (zero beyond
// the grid or on a missing tile, as the reference's void tile), tile 0 is zero.
__global__ void native_to_ref_kernel(const float* __restrict__ nat, float* __restrict__ ref,
                                     const int32_t* __restrict__ tiles, const int32_t* __restrict__ tile_of,
                                     int ntiles, int ny, int nx, int px) {
    const int t = blockIdx.x;
    if (t >= ntiles) return;
    for (int idx = threadIdx.x; idx < 1296; idx += blockDim.x) {
        float v = 0.0f;
        if (t > 0) {
            const int j = tiles[2 * t] * TILE + idx / 36 - 2;
            const int i = tiles[2 * t + 1] * TILE + idx % 36 - 2;
            if (j >= 0 && j < ny && i >= 0 && i < nx && tile_of[(j / TILE) * (nx / TILE) + i / TILE] != 0)
                v = nat[(size_t)(j + GY) * px + i + GX];
        }
        ref[(size_t)t * 1296 + idx] = v;
    }
}

// Tables (ntiles,32,32,rows) and (ntiles,32,32,rows,2) -> level-major pairs and quads (ntiles,rows-1,32,32).
__global__ void pack_tables_kernel(const float* __restrict__ dtab, const float* __restrict__ ftabx,
                                   const float* __restrict__ ftaby, float2* __restrict__ dtab2,
                                   float4* __restrict__ fx, float4* __restrict__ fy, int ntiles, int rows) {
    const size_t n = (size_t)ntiles * (rows - 1) * TILE2;
    for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += (size_t)gridDim.x * blockDim.x) {
        const size_t local = o % TILE2;
        const size_t r = (o / TILE2) % (rows - 1);
        const size_t t = o / ((size_t)TILE2 * (rows - 1));
        const size_t cell = t * TILE2 + local;
        dtab2[o] = make_float2(dtab[cell * rows + r], dtab[cell * rows + r + 1]);
        const float* a = ftabx + cell * rows * 2 + 2 * r;
        fx[o] = make_float4(a[0], a[1], a[2], a[3]);
        const float* b = ftaby + cell * rows * 2 + 2 * r;
        fy[o] = make_float4(b[0], b[1], b[2], b[3]);
    }
}

// The flags of the active list's tiles (is_act). One CTA; a list entry outside the tiles is passed over.
__global__ void __launch_bounds__(1024) active_flags_kernel(StepArgs A, int n) {
    for (int t = threadIdx.x; t < A.ntiles; t += blockDim.x) A.is_act[t] = 0;
    __syncthreads();
    for (int a = threadIdx.x; a < n; a += blockDim.x) {
        const int t = A.active[a];
        if (t >= 0 && t < A.ntiles) A.is_act[t] = 1;
    }
}

// Boundary marks: clear, then one bit per boundary cell; and whether some of them follows another.
__global__ void bmark_kernel(StepArgs A, int clear_words) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t* mark = const_cast<uint32_t*>(A.bmark);
    int32_t* follow = follow_flag(A.ctl);
    if (clear_words > 0) {
        if (tid == 0) *follow = 0;
        for (int w = tid; w < clear_words; w += gridDim.x * blockDim.x) mark[w] = 0u;
        return;
    }
    for (int m = tid; m < A.nb; m += gridDim.x * blockDim.x) {
        const int fid = fid_of_native(A, A.bcell[m]);
        if (A.bkind[m] > 1) *follow = 1;
        atomicOr(mark + fid / TILE, 1u << (fid % TILE));
    }
}

#endif  // W2B_FAST

}  // namespace w2b
