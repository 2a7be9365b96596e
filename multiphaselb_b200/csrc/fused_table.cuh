// fused_table.cuh -- time steps in two or three kernels on any neighbour table.
//
// The operator path runs some fifteen kernels a step (multiPhasePP.c:163-240):
// every population is read and written by the collision and again by the
// streaming, then read by the sums and the velocity, the boundary patches are
// launched one by one, and the interaction force evaluates the EOS nine times
// per node.  Here a step is
//
//   k_table_sum:     pull f*_n, g*_n through the table, boundary program, rho_n,
//                    sum g''_n, and once per node psi_n and 1/rho_n
//   k_table_heat:    (myMRT only) S_n, T_n = sum g'' + S_n / 2, psi_n
//   k_table_finish:  pull again, heat source, Fi, Ft, U_n, collide -> f*_{n+1},
//                    g*_{n+1}
//
// with the state of the fused path between steps (fused.cuh: post-collision
// populations in the two buffers in turn, T and U double-buffered, S).  Pulling
// twice costs less than writing the streamed populations out and reading them
// back.  The reference's state after the last step is rebuilt by the finish
// kernel in EMIT mode.  Lattices this takes: an updated flow, bounce-back, fixedT
// and periodic patches whose order cannot be observed; the others keep the
// operators.  Arithmetic per node is the shared code, so results are
// bit-identical to the operators.
//
// Bound by the latency of the two dependent loads of a pull (table, then
// population): the D2Q9 kernels ask for 8 and 6 blocks of 128 threads per SM,
// the best of 8 to 12 and 5 to 8; the allocator alone takes 101 registers for
// the rare fixedT nodes and runs 4 (49 us).  B200, us per step, thermal channel
// around a cylinder: 768 x 384 127 -> 41, myMRT 137 -> 44, 80 x 70 78 -> 13.5.
#pragma once

#include "fused.cuh"

namespace mplb {

enum TableHeat { TABLE_NONE = 0, TABLE_LITEMP = 1, TABLE_MY = 2 };

struct TableArgs {
    const int32_t* nb;   // pull table [k][n], -1 = missing
    const uint8_t* onb;  // node misses a neighbour
    const double* fin;
    double* fout;
    const double* gin;
    double* gout;
    const double* Told;
    double* Tnew;
    const double* Uold;
    double* Unew;
    double* S;
    double* rho;
    double* psi;  // scratch: psi_n, 1/rho_n of every node
    double* inv;
    double* Fi;  // EMIT outputs
    double* Ft;
    const uint8_t* bcmap;  // as FusedArgs
    double Twall[MPLB_MAX_PATCHES];
    BCProg prog[FUSED_MAX_PROGS];
};

// Populations of node id streamed from `in`; bit k of the result: no source.
template <class L>
__device__ __forceinline__ uint32_t table_pull(const TableArgs& A, uint32_t n, uint32_t id, const double* in, double* v) {
    uint32_t miss = 0;
#pragma unroll
    for (int k = 0; k < L::Q; k++) {
        const int32_t s = __ldg(A.nb + (size_t)k * n + id);
        miss |= (uint32_t)(s == -1) << k;
        v[k] = __ldg(in + (size_t)k * n + (s != -1 ? (uint32_t)s : id));
    }
    return miss;
}

template <class L>
__device__ __forceinline__ void table_flow(const TableArgs& A, uint32_t n, uint32_t id, int pi, double* f) {
    const uint32_t miss = table_pull<L>(A, n, id, A.fin, f);
    if (pi) {
        const BCProg& pr = A.prog[pi];
        for (int o = 0; o < pr.nf; o++) bounce_back<L>(miss, f);
    }
}

template <class L, int GM>
__device__ __forceinline__ void table_heat_pull(const Params& P, const TableArgs& A, uint32_t n, uint32_t id,
                                                int pi, double* g) {
    const uint32_t miss = table_pull<L>(A, n, id, A.gin, g);
    if (!pi) return;
    const BCProg& pr = A.prog[pi];
    for (int o = 0; o < pr.ng; o++) {
        if (pr.gt[o] == MPLB_BC_BOUNCEBACK) {
            bounce_back<L>(miss, g);
            continue;
        }
        // fixedT.c:119-200: the inner neighbour's streamed population (no boundary
        // op writes it: checked on the host) and its U, T of the step before
        const double Tw = A.Twall[pr.gp[o]];
#pragma unroll
        for (int k = 0; k < L::Q; k++) {
            if (!((miss >> k) & 1u)) continue;
            const int32_t m = A.nb[(size_t)revk<L>(k) * n + id];
            if (m == -1) continue;
            const int32_t s = A.nb[(size_t)k * n + (uint32_t)m];
            const double gm = A.gin[(size_t)k * n + (s != -1 ? (uint32_t)s : (uint32_t)m)];
            double eq_nb, eq_bnd;
            if constexpr (GM == TABLE_MY) {
                const double u[3] = {A.Uold[m], A.Uold[(size_t)n + m], L::D == 3 ? A.Uold[2 * (size_t)n + m] : 0.0};
                eq_nb = eq_my_k<L>(P, k, A.Told[m], u);
                eq_bnd = eq_my_k<L>(P, k, Tw, u);
            } else {
                const double u0 = A.Uold[m], u1 = A.Uold[(size_t)n + m];
                eq_nb = eq_heat_k(P, k, A.Told[m], u0, u1);
                eq_bnd = eq_heat_k(P, k, Tw, u0, u1);
            }
            g[k] = eq_bnd + (gm - eq_nb);
        }
    }
}

__device__ __forceinline__ int table_program(const TableArgs& A, uint32_t id) { return A.bcmap ? A.bcmap[id] : 0; }

// Gradients of T_{n-1} and 1/rho_n (their dot product) and divergence of
// U_{n-1}, one-sided at missing neighbours (finiteDifference/*.c).
template <class L>
__device__ __forceinline__ void table_gradients(const TableArgs& A, uint32_t n, uint32_t id, double& dot, double& div) {
    double gT[3] = {0, 0, 0}, gR[3] = {0, 0, 0};
    dot = div = 0;
    const double t = A.Told[id], r = A.inv[id];
#pragma unroll
    for (int d = 0; d < L::D; d++) {
        const int32_t a = A.nb[(size_t)fda<L>(d) * n + id], b = A.nb[(size_t)fdb<L>(d) * n + id];
        const uint32_t ia = a != -1 ? (uint32_t)a : id, ib = b != -1 ? (uint32_t)b : id;
        gT[d] = fd_pair(a, b, A.Told[ia], A.Told[ib], t).v;
        gR[d] = fd_pair(a, b, A.inv[ia], A.inv[ib], r).v;
        const FD u = fd_pair(a, b, A.Uold[(size_t)d * n + ia], A.Uold[(size_t)d * n + ib], A.Uold[(size_t)d * n + id]);
        if (u.present) div += u.v;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) dot += gT[k] * gR[k];
}

template <class L, int GM>
__global__ void __launch_bounds__(128, L::Q == 9 || GM == TABLE_NONE ? 8 : 4) k_table_sum(Params P, TableArgs A) {
    step_dependency_wait();
    const uint32_t n = P.n, id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    const int pi = table_program(A, id);
    double v[L::Q], rho = 0, T = 0;
    table_flow<L>(A, n, id, pi, v);
#pragma unroll
    for (int k = 0; k < L::Q; k++) rho += v[k];
    A.rho[id] = rho;
    if constexpr (GM == TABLE_NONE) {
        T = A.Told[id];
    } else {
        table_heat_pull<L, GM>(P, A, n, id, pi, v);
#pragma unroll
        for (int k = 0; k < L::Q; k++) T += v[k];
        A.Tnew[id] = T;
        A.inv[id] = rcp_rn(rho);
    }
    if constexpr (GM != TABLE_MY) A.psi[id] = potential(P, rho, T);
}

// myMRT: S_n, T_n and psi_n (Tnew holds sum g''_n).
template <class L>
__global__ void __launch_bounds__(128) k_table_heat(Params P, TableArgs A) {
    step_dependency_wait();
    const uint32_t n = P.n, id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    double dot, div;
    table_gradients<L>(A, n, id, dot, div);
    const double rho = A.rho[id];
    const EosRho er = eos_rho(P, rho);
    const double S = heat_source_value_my_er(P, er, rho, A.inv[id], A.Told[id], dot, div);
    const double T = A.Tnew[id] + 0.5 * S;
    A.S[id] = S;
    A.Tnew[id] = T;
    A.psi[id] = potential_p(P, rho, p_eos_at(P, er, rho, T));
}

template <class L, int GM, bool EMIT, bool ST>
__global__ void __launch_bounds__(128, L::Q == 9 ? 6 : (GM == TABLE_NONE ? 5 : 3)) k_table_finish(Params P, TableArgs A) {
    step_dependency_wait();
    const uint32_t n = P.n, id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    const int pi = table_program(A, id);
    const bool onb = A.onb[id] != 0;
    const double rho = A.rho[id], psi = A.psi[id], rr = GM == TABLE_NONE || EMIT ? rcp_rn(rho) : A.inv[id];
    double heat = 0;
    if constexpr (GM == TABLE_LITEMP && !EMIT) {
        double dot, div;
        table_gradients<L>(A, n, id, dot, div);
        heat = heat_source_value_er(P, eos_rho(P, rho), rho, rr, A.Told[id], dot, div, A.S[id]);
    }
    if constexpr (GM == TABLE_MY) heat = A.S[id];
    double f[L::Q], lv[L::D], Fi[3], Ft[3], U[3];
    table_flow<L>(A, n, id, pi, f);
    momentum<L>(f, lv);
    auto nbpsi = [&](int k) { return __ldg(A.psi + A.nb[(size_t)revk<L>(k) * n + id]); };
    force_velocity<L, EMIT>(P, onb, lv, rho, rr, psi, nbpsi, Fi, Ft, U);
    if constexpr (EMIT) {
#pragma unroll
        for (int k = 0; k < L::Q; k++) A.fout[(size_t)k * n + id] = f[k];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            A.Fi[(size_t)j * n + id] = Fi[j];
            A.Ft[(size_t)j * n + id] = Ft[j];
            A.Unew[(size_t)j * n + id] = U[j];
        }
    } else {
        auto term = [&](double* m) {
            if constexpr (ST) {
                if (!onb) {
                    double C[L::Q];
                    surface_tension<L>(P, psi, nbpsi, C);
#pragma unroll
                    for (int k = 0; k < L::Q; k++) m[k] = m[k] + C[k];
                }
            }
        };
        if constexpr (L::Q == 9) collide_limrt_psi<true>(P, f, rho, U, Ft, Fi, psi, term);
        else collide_xumrt_psi<true>(P, f, rho, U, Fi, psi, term);
#pragma unroll
        for (int k = 0; k < L::Q; k++) A.fout[(size_t)k * n + id] = f[k];
    }
    if constexpr (GM != TABLE_NONE) {
        table_heat_pull<L, GM>(P, A, n, id, pi, f);
        if constexpr (!EMIT) {
            const double T = A.Tnew[id];
            if constexpr (GM == TABLE_MY) collide_mymrt<L>(P, f, T, U, heat);
            else if constexpr (L::Q == 9) collide_litemp<true>(P, f, T, U[0], U[1], heat);
            A.S[id] = heat;
#pragma unroll
            for (int j = 0; j < L::D; j++) A.Unew[(size_t)j * n + id] = U[j];
        }
#pragma unroll
        for (int k = 0; k < L::Q; k++) A.gout[(size_t)k * n + id] = f[k];
    }
}

}  // namespace mplb
