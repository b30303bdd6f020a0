// stage_sweep64.cuh -- the plain FP64 form's RK stage for 16x16 and 8x8
// patches as a row sweep: one warp per 16x16 quadrant (two per warp for
// 8x8), no block-wide barriers.
//
// It produces the same bits as stage_kernel<n, ..., FP64> and therefore as
// the reference: the same flux code (flux_roe_2d, flux_2d_module.F90:63-182,
// on records made by the flux's own expressions; boundary flux
// bc_2d_module.F90:14-75), interior face normals and sub-cell volumes from
// the same bilinear nodes (bilinear_node_2d_module.F90:14-36,
// solver_residual_subgrid_2d_module.F90:82-163), edge normals from cell_h
// of the side's level, and each cell's residual summed in the reference's
// order (physics_rhs_structured.c:73-276: the edge faces first, in face_info
// order, a coarse hanging edge's two fluxes one after the other; then
// solver_residual_subgrid_2d's interior faces -F(x-1/2) +F(x+1/2) -F(y-1/2)
// +F(y+1/2)), divided by the volume and negated, then the stage update with
// the reference's coefficients (rk_time_integrators.c). This translation
// unit is compiled with -fmad=false, so no multiply-add is contracted.
//
//   lane = (sub, h, i): quad sub of the warp's 32/(2N) quads, column i,
//        rows R*h .. R*h+R-1 with R = N/2.
//   edges   each lane evaluates one edge face per round (sides 0/1, then
//           2/3; a coarse hanging edge also its second, index-paired flux)
//           into a per-warp table, and the faces between rows R-1 and R;
//   sweep   at step t lane (i, h) takes cell (i, j = Rh+t): its record, the
//           y-face flux at j-1/2 with the record of row j-1, which completes
//           row j-1 (its update is written), then the x-face at i-1/2 with
//           the left neighbour's record taken by a warp shuffle (the flux
//           goes to lane i-1, which needs it as its i+1/2 face, by a second
//           shuffle).
//
// Registers are the limit of an FP64 flux kernel (a flux evaluation holds
// about 60 live doubles), so what a lane carries from one row to the next --
// row j-1's record (its first four values are the input state), partial
// residual and volume -- waits in shared memory, and so does the y-face flux
// while the x-face is evaluated; the row's own-cell inputs (the next row's
// state, the stage's auxiliary inputs) arrive there by cp.async one step
// ahead of use. What a lane needs of its quad's descriptor in every row (the
// signs and order of its edge contributions, the corners) is read once per
// item into a register of flags and shared memory: read from global memory
// row by row it was a third of the warps' waiting.
//
// Bound by the FP64 pipe's latency at 12 warps per SM (168 registers, no
// spills; 128 registers and 16 warps spill 84-212 bytes a thread and are 3%
// slower). 1024^2 cells in 16x16 patches, RK3, one session alone: 356 us per
// step with IEEE division and square root inline, 249 us with this file's
// arithmetic (flux_fp64.cuh) and order; with three sessions' streams
// overlapping 309 -> 187 us per step. That is for domains on which every
// interior normal lies along its axis (roe_flux_any); elsewhere 380 -> 312 us.
#pragma once

#include "async_copy.cuh"
#include "flux_fp64.cuh"
#include "stage_kernel.cuh"
#include "sweep_common.cuh"

namespace amrgpu {

// Dynamic shared memory of the FP64 sweep, in doubles per warp.
template <int N>
struct Sweep64Smem {
    static constexpr int QPW = 32 / (2 * N);
    static constexpr int RS = 9;                      // record: rho, rho u, rho v, rho E, u, v, p, H, sqrt(rho)
    static constexpr int edge = QPW * 4 * 2 * N * 4;  // [quad][side][first/second flux][position][field]
    static constexpr int mid = QPW * N * 4;           // [quad][column][field]: faces between rows R-1 and R
    static constexpr int carry = (RS + 4 + 1) * 32;   // [record, partial / y-face flux, volume][lane]
    static constexpr int qbuf = 4 * 32;               // next row's state [field][lane]
    static constexpr int abuf = 8 * 32;               // auxiliary inputs a0, a1 [field][lane]
    static constexpr int corner = QPW * 8;            // the quad's corners
    static constexpr int col0 = QPW * (N + 2) * 2;    // bilinear nodes (0, row), row = 0..N
    static constexpr int o_edge = 0, o_mid = o_edge + edge, o_carry = o_mid + mid, o_q = o_carry + carry,
                         o_a = o_q + qbuf, o_corner = o_a + abuf, o_col0 = o_corner + corner;
    static constexpr int per_warp = o_col0 + col0;
    static constexpr size_t bytes(int warps) { return sizeof(double) * (size_t)per_warp * (size_t)warps; }
};

// ST = 0: any scheme and stage, read from the arguments; ST = 1..3: stage
// ST of the reference's RK3 (the FP64 form's default scheme) fixed at
// compile time -- the same update expressions without the per-cell switch.
template <int N, int WARPS, int ST>
__device__ __forceinline__ void sweep64_body(const StageArgs &a)
{
    static_assert(N == 16 || N == 8, "row sweep for 16x16 and 8x8 patches");
    using S = Sweep64Smem<N>;
    constexpr int NN = N * N;
    constexpr int QPW = S::QPW;
    constexpr int R = N / 2;  // rows per half-patch
    constexpr int RS = S::RS;
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) double sm64[];
    __shared__ double red[64];
    __shared__ int s_last;

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int sub = lane / (2 * N), l = lane % (2 * N);
    const int i = l % N, h = l / N;
    const long long stride = a.stride;
    const double scale_factor = 2.0 / (double)N;
    const double xi1 = scale_factor * (double)(i + 1) - 1.0;  // nodes at column i+1

    double *wsm = sm64 + (size_t)w * S::per_warp;
    double(*sedge)[4][2][N][4] = reinterpret_cast<double(*)[4][2][N][4]>(wsm + S::o_edge);
    double(*smid)[N][4] = reinterpret_cast<double(*)[N][4]>(wsm + S::o_mid);
    double *car = wsm + S::o_carry + lane;  // slot c at car[32 c]
    double *qb = wsm + S::o_q + lane;       // field f at qb[32 f]
    double *ab = wsm + S::o_a + lane;       // a0 field f at ab[32 f], a1 at ab[32 (4 + f)]
    double *g = wsm + S::o_corner + 8 * sub;
    double *c0 = wsm + S::o_col0 + 2 * (N + 2) * sub;  // node (0, row) at c0[2 row]
    enum { kPart = RS, kVol = RS + 4 };

    const double dt = sweep_step_dt(a);
    double my_dt_min = a.dt_cap;
    double my_norm = 0.0;
    int my_flags = 0;
    // the reference RK3's auxiliary inputs: none in stage 1, Q0 and k1 in
    // stage 2, the combination C in stage 3
    const bool has_a0 = ST > 0 ? ST >= 2 : a.a0 != nullptr;
    const bool has_a1 = ST > 0 ? ST == 2 : a.a1 != nullptr;

    // work items as in the FP32 sweep: first by warp index, then from the
    // quad counter; a quad past the end is computed on the item's first
    // quad and neither stored nor reduced
    const int nwarps = gridDim.x * WARPS;
    const int nitems = (a.nquad + QPW - 1) / QPW;
    int item = blockIdx.x * WARPS + w;
    while (item < nitems) {
        const bool valid = QPW == 1 || item * QPW + sub < a.nquad;
        const int quad = valid ? item * QPW + sub : item * QPW;
        const QuadDesc &qd = a.quads[quad];
        const double *Qq = a.qin + (long long)quad * NN;
        auto load_rec = [&](const double *base, int cell, double P[RS]) {
            double q[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) q[f] = base[f * stride + cell];
            cell_prims_fp64(q, P);
        };
        // the first row's state, on its way while the edges are computed
#pragma unroll
        for (int f = 0; f < 4; ++f) cp_async8(qb + 32 * f, Qq + f * stride + (R * h) * N + i);
        cp_async_commit();
        cp_async_commit();  // (no auxiliary group before the first row)
        if (l < 8) g[l] = qd.corner[l];
        // what the rows need of the sides, as bits: this lane's corner takes
        // its y-side's contribution before its x-side's (bit 0: bottom,
        // bit 1: top), side s adds its flux (bit 2 + s; else subtracts it),
        // side s is a coarse hanging edge (bit 6 + s)
        unsigned flags = 0;
        {
            const int sx = i == 0 ? 0 : 1;
            const int rx = qd.side[sx].rank;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int kind = qd.side[s].kind;
                if (kind == kSideBoundary || (s & 1)) flags |= 4u << s;
                if (kind == kSideCoarseHang) flags |= 64u << s;
                if (s >= 2 && qd.side[s].rank < rx) flags |= 1u << (s - 2);
            }
        }
        __syncwarp();
        // the nodes of column 0 (lanes 0..N of a quad's 2N: lane l row l)
        if (l <= N) bilinear_node(g, -1.0, scale_factor * (double)l - 1.0, c0[2 * l], c0[2 * l + 1]);

        // ---------------- edges: round 0 sides 0 / 1, round 1 sides 2 / 3
#pragma unroll 1
        for (int round = 0; round < 2; ++round) {
            const int s = 2 * round + h, m = i;
            const bool xd = round == 0;
            const SideDesc d = qd.side[s];
            const int own = (s == 0) ? m * N : (s == 1) ? m * N + N - 1 : (s == 2) ? m : (N - 1) * N + m;
            double Po[RS], fl[4];
            load_rec(Qq, own, Po);
            const double hc = cell_h_of(a.h_base, d.level, N);
            if (d.kind == kSideBoundary) {
                const double n0 = xd ? ((s & 1) ? hc : -hc) : 0.0;
                const double n1 = xd ? 0.0 : ((s & 1) ? hc : -hc);
                bc_flux_fp64(d.bc, Po, n0, n1, a.qinflow, fl);
#pragma unroll
                for (int f = 0; f < 4; ++f) sedge[sub][s][0][m][f] = fl[f];
            } else {
                // the neighbour's facing cell at the same position (a coarse
                // hanging edge pairs it with both fine quads)
                const int fc = facing_cell<N>(s, m);
                const int nk = (d.kind == kSideCoarseHang) ? 2 : 1;
                const double n0 = xd ? hc : 0.0, n1 = xd ? 0.0 : hc;
#pragma unroll 1
                for (int k = 0; k < nk; ++k) {
                    double Pn[RS], Lr[RS], Rr[RS];
                    load_rec(a.qin + (long long)(k == 0 ? d.nbr0 : d.nbr1) * NN, fc, Pn);
#pragma unroll
                    for (int c = 0; c < RS; ++c) {
                        Lr[c] = (s & 1) ? Po[c] : Pn[c];
                        Rr[c] = (s & 1) ? Pn[c] : Po[c];
                    }
                    roe_flux_prim_fp64<2>(Lr, Rr, n0, n1, fl);
#pragma unroll
                    for (int f = 0; f < 4; ++f) sedge[sub][s][k][m][f] = fl[f];
                }
            }
        }
        // ---------------- the faces between rows R-1 and R (column i):
        // normal from the nodes (i+1, R) and (i, R)
        {
            double P[RS], O[RS], fl[4];
            load_rec(Qq, (R - 1 + h) * N + i, P);
#pragma unroll
            for (int c = 0; c < RS; ++c) O[c] = __shfl_xor_sync(FULL, P[c], N);
            if (h == 0) {
                const double eta = scale_factor * (double)R - 1.0;
                double x1, y1, x2, y2;
                bilinear_node(g, xi1, eta, x1, y1);
                bilinear_node(g, scale_factor * (double)i - 1.0, eta, x2, y2);
                roe_flux_prim_fp64<1>(P, O, y2 - y1, x1 - x2, fl);
#pragma unroll
                for (int f = 0; f < 4; ++f) smid[sub][i][f] = fl[f];
            }
        }
        __syncwarp();

        // the edge contributions of cell (i, j) in face_info order, starting
        // from 0 (physics_rhs_structured.c:73-262 visits faces in order)
        auto edge_sum = [&](int j, double r[4]) {
            const int sx = (i == 0) ? 0 : (i == N - 1) ? 1 : -1;
            const int sy = (j == 0) ? 2 : (j == N - 1) ? 3 : -1;
            if (sx < 0 && sy < 0) return;
            int first = sx, second = sy;
            if (sx >= 0 && sy >= 0 && (flags >> (sy - 2) & 1u)) {
                first = sy;
                second = sx;
            }
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int s = pass == 0 ? first : second;
                if (s < 0) continue;
                const int m = (s < 2) ? j : i;
                const bool hang = flags >> (6 + s) & 1u;
                const double *F = sedge[sub][s][0][m];
                const double *F2 = sedge[sub][s][1][m];
                if (flags >> (2 + s) & 1u) {
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        r[f] = r[f] + F[f];
                        if (hang) r[f] = r[f] + F2[f];
                    }
                } else {
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        r[f] = r[f] - F[f];
                        if (hang) r[f] = r[f] - F2[f];
                    }
                }
            }
        };
        // finishes row jr from the carried state: + F(y+1/2) when that face
        // is interior, / volume, x -1, stage update with the auxiliary
        // inputs in ab, last-stage reductions
        auto finish = [&](int jr, const double *gup) {
            const long long gi = (long long)quad * NN + jr * N + i;
            const double vol = car[32 * kVol];
            double r[4], kv[4], qn[4], q0v[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const double p = car[32 * (kPart + f)];
                r[f] = gup ? p + gup[f] : p;
                q0v[f] = car[32 * f];
            }
            residual_rate(r, vol, kv);
            if (!valid) return;
            auto A0 = [&](int f) -> double { return ab[32 * f]; };
            auto A1 = [&](int f) -> double { return ab[32 * (4 + f)]; };
            if constexpr (ST > 0) rk_update<kSchemeRK3, ST>(a, dt, stride, gi, q0v, kv, A0, A1, qn);
            else rk_update(a, dt, stride, gi, q0v, kv, A0, A1, qn);
            if (ST > 0 ? ST == 3 : a.last_stage != 0) {
#pragma unroll
                for (int f = 0; f < 4; ++f) my_norm += kv[f] * kv[f];
                if (a.cfl_on) {
                    const double cand = cfl_candidate_fp64(qn, vol, a.cfl);
                    if (cand < my_dt_min) my_dt_min = cand;
                }
                const double rho = qn[0];
                const double pe = qn[3] * rho - 0.5 * (qn[1] * qn[1] + qn[2] * qn[2]);
                if (!(rho > 0.0) || !(pe > 0.0)) my_flags |= kFlagNegative;
            }
        };
        // the auxiliary inputs of row jr into ab (one cp.async group)
        auto fetch_aux = [&](int jr) {
            const long long gi = (long long)quad * NN + jr * N + i;
            if (has_a0) {
#pragma unroll
                for (int f = 0; f < 4; ++f) cp_async8(ab + 32 * f, a.a0 + f * stride + gi);
            }
            if (has_a1) {
#pragma unroll
                for (int f = 0; f < 4; ++f) cp_async8(ab + 32 * (4 + f), a.a1 + f * stride + gi);
            }
            cp_async_commit();
        };

        // ---------------- sweep over the lane's R rows. cp.async groups in
        // flight at the start of step t: the state of row j (issued one step
        // earlier) and the auxiliary inputs of row j-1.
        //
        // node (i+1, row) of the lane, from the corners; node (i, row) is the
        // left lane's, and lane 0's comes from column 0's table
        auto nodes = [&](int row, double &x0, double &y0, double &x1, double &y1) {
            bilinear_node(g, xi1, scale_factor * (double)row - 1.0, x1, y1);
            x0 = __shfl_up_sync(FULL, x1, 1, N);
            y0 = __shfl_up_sync(FULL, y1, 1, N);
            const double ex = c0[2 * row], ey = c0[2 * row + 1];
            x0 = i == 0 ? ex : x0;
            y0 = i == 0 ? ey : y0;
        };
        double xa, ya, xb, yb;  // nodes (i, j) and (i+1, j) of the current row
        nodes(R * h, xa, ya, xb, yb);
#pragma unroll 1
        for (int t = 0; t < R; ++t) {
            const int j = R * h + t;
            cp_async_wait_group<1>();  // row j's state has landed
            double P[RS];
            {
                double q4[4];
#pragma unroll
                for (int f = 0; f < 4; ++f) q4[f] = qb[32 * f];
                cell_prims_fp64(q4, P);
            }
            // the next row's state into the buffer just read (the record
            // above consumed it)
            if (t < R - 1) {
#pragma unroll
                for (int f = 0; f < 4; ++f) cp_async8(qb + 32 * f, Qq + f * stride + (j + 1) * N + i);
            }
            cp_async_commit();
            // y-face at j-1/2, nodes (i+1, j) -> (i, j), row j-1's record:
            // completes row j-1, whose partial residual makes room for it
            if (t > 0) {
                double A[RS], G[4];
#pragma unroll
                for (int c = 0; c < RS; ++c) A[c] = car[32 * c];
                roe_flux_prim_fp64<1>(A, P, ya - yb, xb - xa, G);
                cp_async_wait_group<1>();  // row j-1's auxiliary inputs
                finish(j - 1, G);
#pragma unroll
                for (int f = 0; f < 4; ++f) car[32 * (kPart + f)] = G[f];
            }
            fetch_aux(j);
            // carry row j's record to the next step
#pragma unroll
            for (int c = 0; c < RS; ++c) car[32 * c] = P[c];
            // nodes (i, j+1), (i+1, j+1), the cell's volume and the x-face at
            // i-1/2, nodes (i, j) -> (i, j+1), the left neighbour's record
            // (lane i = 0's is an edge face)
            double n0, n1;
            {
                double xc, yc, xd, yd;
                nodes(j + 1, xc, yc, xd, yd);
                car[32 * kVol] = subcell_volume(xa, ya, xb, yb, xc, yc, xd, yd);
                n0 = yc - ya;
                n1 = xa - xc;
                xa = xc;
                ya = yc;
                xb = xd;
                yb = yd;
            }
            double F[4];
            {
                double A[RS];
#pragma unroll
                for (int c = 0; c < RS; ++c) A[c] = __shfl_up_sync(FULL, P[c], 1, N);
                roe_flux_prim_fp64<0>(A, P, n0, n1, F);
            }
            double Fr[4], r[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) Fr[f] = __shfl_down_sync(FULL, F[f], 1, N);
#pragma unroll
            for (int f = 0; f < 4; ++f) r[f] = 0.0;
            edge_sum(j, r);
            // interior faces only (lane 0's low and lane N-1's high x-face
            // and the quad's low y-face are edge faces, summed above): each
            // sum is formed and kept or dropped by a select, not a branch
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const double rl = r[f] - F[f];
                r[f] = i > 0 ? rl : r[f];
                const double rr = r[f] + Fr[f];
                r[f] = i < N - 1 ? rr : r[f];
                const double G = t > 0 ? car[32 * (kPart + f)] : smid[sub][i][f];
                const double rg = r[f] - G;
                car[32 * (kPart + f)] = t > 0 || h == 1 ? rg : r[f];
            }
        }
        // the half's top row: the face between rows R-1 and R (h = 0) or the
        // patch's top edge, already summed (h = 1)
        cp_async_wait_group<0>();
        finish(R * h + R - 1, h == 0 ? smid[sub][i] : nullptr);
        __syncwarp();  // the next item rewrites this warp's tables
        unsigned nxt = 0;
        if (lane == 0) nxt = atomicAdd(&a.scal->work_next, 1u);
        item = nwarps + (int)__shfl_sync(FULL, nxt, 0);
    }

    sweep_reduce<WARPS>(a, my_dt_min, my_norm, my_flags, red, &s_last);
}

template <int WARPS, int MINB, int ST = 0>
__global__ void __launch_bounds__(WARPS * 32, MINB) sweep64_16_kernel(const StageArgs a)
{
    stage_launch_gate();
    sweep64_body<16, WARPS, ST>(a);
}

template <int WARPS, int MINB, int ST = 0>
__global__ void __launch_bounds__(WARPS * 32, MINB) sweep64_8_kernel(const StageArgs a)
{
    stage_launch_gate();
    sweep64_body<8, WARPS, ST>(a);
}

}  // namespace amrgpu
