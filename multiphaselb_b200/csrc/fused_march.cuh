// fused_march.cuh -- D2Q9 fused step with myMRT heat, one warp per strip of
// columns marching along y.
//
// With myMRT, T_n = sum g'' + S_n / 2 and S_n of a node needs rho_n one node
// further out, so the psi that a node's force takes from its neighbours needs
// rho_n two nodes out.  The tile kernels (fused.cuh) take that from a pre-pass
// that pulls and sums the whole lattice once more.  Here a warp holds 32
// neighbouring columns and walks up its chunk of rows: row j is pulled and
// summed, row j - 1 gets its heat source, T and psi, row j - 2, whose
// neighbourhood is then complete, is finished.  The last three rows' psi,
// 1/rho, T_{n-1} and U_{n-1} lie in rings of the warp's own shared memory.
// The outer H = 2 lanes on either side and H rows before and after the chunk
// are summed only, so a node's moments are computed 32/28 (1 + 4/rows) times
// instead of twice (pre-pass and step) plus a ring of 1.33 to 1.6, and no warp
// waits for another.
//
// Bound by latency and FP64 issue: a warp's next row is requested (cp.async)
// when the stage of the row it finishes has been read, so the copies overlap
// that row's collision.  Shared memory (17.7 KB) and registers leave 12 warps
// per SM.  B200, 1021 x 2039 column, back to back: 201 us a step against
// 294 us of the best tile kernel and its pre-pass; on lattices of a wave or
// less the tile kernels' shorter chain wins (61 x 97: 16 us against 26 us),
// which the tile autotuner finds.  The same march for liTempMRT or without
// heat (H = 1, two rows in flight) measured no gain over the tile kernels: its
// 30-column rows write partial sectors (the tile kernels' are aligned), and
// their ring costs less than myMRT's pre-pass.
//
// Nodes near a wall or with a boundary program (FusedArgs::mx, my: the
// distance from the faces that holds them all) go through pull_node.
// Arithmetic per node is the shared code, so results are bit-identical to the
// other fused kernels.
#pragma once

#include "fused.cuh"

namespace mplb {

constexpr int MARCH_H = 2, MARCH_W = 32 - 2 * MARCH_H;  // halo, and columns a warp owns

// Column (or row) c of an axis, up to two nodes outside the box: wrapped when
// periodic, -1 when absent.
MPLB_HD int march_wrap(int c, int ext, int periodic) {
    if (c < 0) return periodic ? c + ext : -1;
    if (c >= ext) return periodic ? c - ext : -1;
    return c;
}

// Shared memory of a warp: the pulled populations of three rows (each lane's
// own column only), and three-row rings that its neighbour lanes read.
template <bool F_ON>
struct MarchSmem {
    double pop[MARCH_H + 1][F_ON ? 18 : 9][32];
    double psi[F_ON ? 3 : 1][32];
    double inv[3][32];
    double To[3][32];
    double U0[3][32];
    double U1[3][32];
};

// A row's three pull rows (element offsets): below (populations moving up),
// the row itself, above.
struct MarchRow {
    uint32_t dn, at, up;
};
__device__ __forceinline__ MarchRow march_row(const FusedArgs& A, int y) {
    const int yd = march_wrap(y - 1, A.ny, A.py), yu = march_wrap(y + 1, A.ny, A.py);
    MarchRow r;
    r.at = (uint32_t)y * (uint32_t)A.nx;
    r.dn = (uint32_t)(yd >= 0 ? yd : y) * (uint32_t)A.nx;
    r.up = (uint32_t)(yu >= 0 ? yu : y) * (uint32_t)A.nx;
    return r;
}

template <bool F_ON, bool HAS_BC>
__global__ void __launch_bounds__(32, 8) k_march_my_d2q9(Params P, FusedArgs A) {
    step_dependency_wait();
    using L = D2Q9T;
    constexpr int H = MARCH_H, NF = F_ON ? 9 : 0;
    __shared__ MarchSmem<F_ON> s;
    const uint32_t n = P.n;
    const int nx = A.nx, ny = A.ny;
    const int lane = threadIdx.x;
    const int strip = blockIdx.x % A.tiles_x, chunk = blockIdx.x / A.tiles_x;
    const int y0 = chunk * A.zchunk, y1 = min(y0 + A.zchunk, ny);

    // the lane's column, its pull columns, and whether it is near an x face
    const int xo = strip * MARCH_W - H + lane;
    const int xw = xo < nx + H ? march_wrap(xo, nx, A.px) : -1;
    const bool col = xw >= 0;
    const int x = col ? xw : 0;
    const bool own = col && lane >= H && lane < 32 - H && xo < nx, mid = lane >= 1 && lane <= 30;
    const int xl = march_wrap(x - 1, nx, A.px), xr = march_wrap(x + 1, nx, A.px);
    const bool hl = xl >= 0, hr = xr >= 0;
    const uint32_t c0 = (uint32_t)x, cm = (uint32_t)(hl ? xl : x), cp = (uint32_t)(hr ? xr : x);
    const bool near_x = x <= A.mx || x >= nx - 1 - A.mx;

    // request row j: its populations into stage st, T and U of the step before
    // into ring row q
    auto request = [&](int j, int st, int q) {
        const int y = march_wrap(j, ny, A.py);
        if (col && y >= 0) {
            const MarchRow r = march_row(A, y);
            static_for<9>([&](auto kk) {
                constexpr int k = decltype(kk)::value;
                const uint32_t row = cyk<L>(k) == 1 ? r.dn : (cyk<L>(k) == -1 ? r.up : r.at);
                const uint32_t c = cxk<L>(k) == 1 ? cm : (cxk<L>(k) == -1 ? cp : c0);
                if constexpr (F_ON) cp_async8(&s.pop[st][k][lane], A.fin + ((size_t)k * n + row) + c);
                cp_async8(&s.pop[st][NF + k][lane], A.gin + ((size_t)k * n + row) + c);
            });
            cp_async8(&s.To[q][lane], A.Told + r.at + c0);
            cp_async8(&s.U0[q][lane], A.Uold + r.at + c0);
            cp_async8(&s.U1[q][lane], A.Uold + ((size_t)n + r.at) + c0);
        }
        cp_async_commit();
    };

    double rho1 = 0, rr1 = 0, T1 = 0;          // row j - 1
    double rho2 = 0, rr2 = 0, T2 = 0, S2 = 0;  // row j - 2
    bool have1 = false, have2 = false;
    int st = 0;                  // stage of row j
    int qn = 0, qc = 2, qp = 1;  // ring rows of j, j - 1, j - 2 (psi: j - 3, j - 1, j - 2)

    request(y0 - H, 0, 0);
    for (int j = y0 - H; j < y1 + H; j++) {
        // ---- row j has landed: sum it
        cp_async_wait0();
        const int yw = march_wrap(j, ny, A.py);
        const int y = yw >= 0 ? yw : 0;
        const bool near = near_x || y <= A.my || y >= ny - 1 - A.my;
        const bool have = col && yw >= 0;
        const uint32_t id = (uint32_t)y * (uint32_t)nx + c0;
        double rho = 0, T = 0, rr = 0;
        if (have) {
            if (near) {
                double f[9], g[9];
                pull_node<L, F_ON, true, HAS_BC>(P, A, x, y, 0, id, f, g, rho, T);
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    if constexpr (F_ON) s.pop[st][k][lane] = f[k];
                    s.pop[st][NF + k][lane] = g[k];
                }
            } else {
                if constexpr (F_ON) {
#pragma unroll
                    for (int k = 0; k < 9; k++) rho += s.pop[st][k][lane];
                } else {
                    rho = A.rho_c[id];
                }
#pragma unroll
                for (int k = 0; k < 9; k++) T += s.pop[st][NF + k][lane];
            }
            rr = rcp_rn(rho);
            s.inv[qn][lane] = rr;
        }
        __syncwarp();

        // ---- row i = j - 1: heat source, T, psi
        const int i = j - 1;
        double S1 = 0;
        if (have1 && mid && i >= y0 - 1) {
            const double To = s.To[qc][lane];
            double gT[3] = {0, 0, 0}, gR[3] = {0, 0, 0}, dot = 0, div = 0;
            if (x > 0 && x < nx - 1 && i > 0 && i < ny - 1) {  // both neighbours on both axes
                gT[0] = 0.5 * (s.To[qc][lane + 1] - s.To[qc][lane - 1]);
                gR[0] = 0.5 * (s.inv[qc][lane + 1] - s.inv[qc][lane - 1]);
                div += 0.5 * (s.U0[qc][lane + 1] - s.U0[qc][lane - 1]);
                gT[1] = 0.5 * (s.To[qn][lane] - s.To[qp][lane]);
                gR[1] = 0.5 * (s.inv[qn][lane] - s.inv[qp][lane]);
                div += 0.5 * (s.U1[qn][lane] - s.U1[qp][lane]);
            } else {
                // i may lie outside the box by one (wrapped): its own row there
                const int yi = march_wrap(i, ny, A.py);
                const bool hd = A.py || yi > 0, hu = A.py || yi < ny - 1;
                FD t = fd_pair(hr ? 0 : -1, hl ? 0 : -1, s.To[qc][lane + 1], s.To[qc][lane - 1], To);
                FD q = fd_pair(hr ? 0 : -1, hl ? 0 : -1, s.inv[qc][lane + 1], s.inv[qc][lane - 1], rr1);
                FD u = fd_pair(hr ? 0 : -1, hl ? 0 : -1, s.U0[qc][lane + 1], s.U0[qc][lane - 1], s.U0[qc][lane]);
                gT[0] = t.v;
                gR[0] = q.v;
                if (u.present) div += u.v;
                t = fd_pair(hu ? 0 : -1, hd ? 0 : -1, s.To[qn][lane], s.To[qp][lane], To);
                q = fd_pair(hu ? 0 : -1, hd ? 0 : -1, s.inv[qn][lane], s.inv[qp][lane], rr1);
                u = fd_pair(hu ? 0 : -1, hd ? 0 : -1, s.U1[qn][lane], s.U1[qp][lane], s.U1[qc][lane]);
                gT[1] = t.v;
                gR[1] = q.v;
                if (u.present) div += u.v;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) dot += gT[k] * gR[k];
            const EosRho er = eos_rho(P, rho1);
            S1 = heat_source_value_my_er(P, er, rho1, rr1, To, dot, div);
            T1 = T1 + 0.5 * S1;
            // into the ring row that psi of row j - 4 leaves
            if constexpr (F_ON) s.psi[qc][lane] = potential_p(P, rho1, p_eos_at(P, er, rho1, T1));
        }
        __syncwarp();

        // ---- finish row e = j - 2
        const int e = j - H;
        const int se = st == H ? 0 : st + 1;  // stage of row e
        const bool fin = e >= y0 && own && have2;
        double f[9], g[9];
        if (fin) {
#pragma unroll
            for (int k = 0; k < 9; k++) {
                if constexpr (F_ON) f[k] = s.pop[se][k][lane];
                g[k] = s.pop[se][NF + k][lane];
            }
        }
        // row j + 1 into the stage and the ring row that were just read
        if (j + 1 < y1 + H) request(j + 1, se, qp);
        if (fin) {
            const uint32_t ie = (uint32_t)e * (uint32_t)nx + c0;
            const bool onb = (!A.px && (x == 0 || x == nx - 1)) || (!A.py && (e == 0 || e == ny - 1));
            double psi = 0;
            if constexpr (F_ON) psi = s.psi[qp][lane];
            // psi ring rows of e - 1, e, e + 1: qn, qp, qc
            auto nbpsi = [&](int k) {
                return s.psi[cyk<L>(k) == 0 ? qp : (cyk<L>(k) == 1 ? qc : qn)][lane + cxk<L>(k)];
            };
            finish_node<L, F_ON, true, false, decltype(nbpsi), true>(P, A, ie, onb, f, g, rho2, rr2, T2, psi, nbpsi, S2);
        }
        __syncwarp();  // the ring row of psi that row j takes next has been read
        st = se;
        const int q = qp;
        qp = qc;
        qc = qn;
        qn = q;
        rho2 = rho1;
        rr2 = rr1;
        T2 = T1;
        S2 = S1;
        have2 = have1;
        rho1 = rho;
        rr1 = rr;
        T1 = T;
        have1 = have;
    }
}

// Launch geometry: strips of MARCH_W columns; the chunk count whose blocks (one
// warp each, `resident` of them at once on the device) waste the fewest slots.
inline Geom march_geometry(const FusedArgs& A, int resident) {
    Geom g;
    g.tiles_x = (A.nx + MARCH_W - 1) / MARCH_W;
    g.tiles_y = 1;
    int best = 1;
    double best_t = 1e30;
    for (int c = 1; c <= std::max(1, A.ny / 4); c++) {
        const int rows = (A.ny + c - 1) / c;
        const long blocks = (long)g.tiles_x * ((A.ny + rows - 1) / rows);
        const double t = (double)((blocks + resident - 1) / resident) * (rows + MARCH_H);
        if (t < best_t - 1e-9) {
            best_t = t;
            best = c;
        }
    }
    g.zchunk = (A.ny + best - 1) / best;
    g.nblocks = g.tiles_x * ((A.ny + g.zchunk - 1) / g.zchunk);
    return g;
}

}  // namespace mplb
