// fused_tma.cuh -- D3Q15 fused step with the plane neighbourhood staged by TMA.
//
// The same time step as k_fused_d3q15 (pull-stream, moments, psi on the tile
// and a one-node ring, force, velocity, xuMRT collision: lbstream.c:16-62,
// xuMRTDensity.c, potential.c:7-13, interactionForce.c:47-79,
// xuMRTVelocity.c:19-44, xuMRTCollision.c:46-89), for fully periodic boxes
// without boundary programs (the static-bubble workloads).  What differs is
// how a plane reaches the block:
//
//   * for every population k the tile's pull sources on plane z - c_kz form
//     one box of (TX+4) x (TY+2) nodes starting at x0-2, y0-1-c_ky (x0-2 is
//     even, so the box starts on a 16-byte boundary), and the temperature
//     plane one more box: 16 boxes per plane, each one TMA tensor copy
//     (cp.async.bulk.tensor, no multicast) into shared memory, completing on
//     the plane's mbarrier;
//   * a tile on a face of the box needs the periodic images of what lies
//     outside, which a tensor copy fills with zeros: one plane later, when the
//     copies have landed, some of its threads write those columns with 16-byte
//     cp.async and those rows with bulk copies (patch_wrapped), completing on a
//     second mbarrier;
//   * two stages: plane p+2 is requested as soon as plane p's stage has been
//     read (after the plane barrier), so its copies overlap two planes of
//     collisions.  The own node's pulled populations are carried in
//     registers from the plane they were read on to the collision one plane
//     later, so a stage is free once its psi pass is done.
//
// Per plane: wait for the stage, psi of every tile and ring slot (the sums
// in k order as pull_node), one barrier, request plane p+2, collide plane
// p-1 (the shared node arithmetic).  psi lives in a four-plane ring so one
// barrier per plane suffices.  The ring's slots fall to the first warps, so
// the barrier is split: a warp arrives once its psi is written, transforms
// its nodes' populations of plane p-1 to moments (a quarter of the
// arithmetic, which needs no neighbour), and only then waits.  Results are
// bit-identical to the other fused kernels.
//
// What set the time was the face tiles: every tile of a 192^3 lattice runs at
// once, and tiles on a face used to copy each of a plane's 160 rows with one or
// two bulk copies, which the copy engine starts every 30 cycles or so (9,300
// cycles a plane where a tile of tensor copies needs 6,700).  B200, 192^3, us a
// step: 480 before, 390 now; 345 with tensor copies alone (wrong at the faces).
//
// Every wait on an mbarrier is bounded: on a timeout the kernel records
// MPLB_KERR_WAIT in A.kerr, waits (bounded again) for the copies it issued
// and returns; the host reports MPLB_E_TIMEOUT at the next synchronising
// call.
#pragma once

#include <cuda.h>

#include "fused.cuh"
#include "tma_util.cuh"

namespace mplb {

template <int TX, int TY>
struct TmaTile {
    static constexpr int BX = TX + 4, BY = TY + 2;  // box extent: x from x0-2, y from y0-1-c_y
    static constexpr int BOX_BYTES = BX * BY * 8;
    static constexpr int BOX_PITCH = (BOX_BYTES + 127) / 128 * 128;  // each box at a 128-byte boundary
    static constexpr int NBOX = 16;                                   // 15 populations + T
    static constexpr int STAGE_BYTES = NBOX * BOX_PITCH;
    static constexpr int NSTAGE = 2;
    static constexpr int EX = TX + 2, EY = TY + 2;  // tile + ring
    static constexpr int NPSI = 4;                  // psi planes kept
    static constexpr int HEAD = 128;                // mbarriers (stages, psi planes), failure flag
    static constexpr size_t SMEM = 128 /* base alignment slack */ + HEAD + (size_t)NSTAGE * STAGE_BYTES +
                                   (size_t)NPSI * EY * EX * 8;
    static_assert(BX * 8 % 16 == 0, "box rows must be whole 16-byte units");
    static_assert(TX % 2 == 0, "x0 - 2 must be even");
};

// finish_node for a node of a fully periodic isothermal D3Q15 lattice whose
// populations are already moments (m = M f; m[0] is not used): moments 3, 5
// and 7 are its momentum, summed in the order of momentum().
template <bool ST, class PsiAt>
__device__ __forceinline__ void finish_moments(const Params& P, const FusedArgs& A, uint32_t id, double* m, double rho,
                                               double rr, double psi, PsiAt nbpsi) {
    using L = D3Q15T;
    if (id - A.own_lo >= A.own_cnt) return;
    double Fi[3], Ft[3], U[3], f[15];
    const double lv[3] = {m[3], m[5], m[7]};
    force_velocity<L, false>(P, false, lv, rho, rr, psi, nbpsi, Fi, Ft, U);
    auto term = [&](double* v) {
        if constexpr (ST) {
            double C[15];
            surface_tension<L>(P, psi, nbpsi, C);
#pragma unroll
            for (int k = 0; k < 15; k++) v[k] = v[k] + C[k];
        }
    };
    relax_xumrt<true>(P, m, f, rho, U, Fi, psi, term);
#pragma unroll
    for (int k = 0; k < 15; k++) A.fout[(size_t)k * P.n + id] = f[k];
    for (int q = 0; q < A.nmirror; q++) {
        const MirrorRange& M = A.mirror[q];
        if (id - M.lo >= M.cnt) continue;
        const size_t d = (size_t)M.dst + (id - M.lo), nd = M.n_dst;
#pragma unroll
        for (int k = 0; k < 15; k++) M.f[(size_t)k * nd + d] = f[k];
    }
}

template <int TX, int TY, int MINB, bool ST = false>
__global__ void __launch_bounds__(TX * TY, MINB)
    k_fused_d3q15_tma(Params P, FusedArgs A, const __grid_constant__ CUtensorMap tm_f,
                      const __grid_constant__ CUtensorMap tm_T) {
    step_dependency_wait();
    using L = D3Q15T;
    using G = TmaTile<TX, TY>;
    constexpr int NT = TX * TY, EX = G::EX, EY = G::EY, NRING = 2 * EX + 2 * TY;
    extern __shared__ unsigned char dsm_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)dsm_raw + 127) & ~(uintptr_t)127);
    uint64_t* bar = reinterpret_cast<uint64_t*>(base);
    uint64_t* face_bar = bar + G::NSTAGE;  // face tiles: the wrapped parts of a stage
    uint64_t* psi_bar = face_bar + G::NSTAGE;
    volatile int* s_fail = reinterpret_cast<volatile int*>(psi_bar + 1);
    unsigned char* stage0 = base + G::HEAD;
    double(*s_psi)[EY][EX] = reinterpret_cast<double(*)[EY][EX]>(stage0 + G::NSTAGE * G::STAGE_BYTES);

    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    const int tiles = A.tiles_x * A.tiles_y;
    const int col = blockIdx.x % tiles, chunk = blockIdx.x / tiles;
    const int x0 = (col % A.tiles_x) * TX, y0 = (col / A.tiles_x) * TY;
    const int z0 = chunk * A.zchunk, z1 = min(z0 + A.zchunk, A.nz);
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    const uint32_t n = P.n;
    // a tile on a periodic face: parts of its boxes lie outside the lattice
    const bool face = x0 == 0 || x0 + TX == nx || y0 == 0 || y0 + TY == ny;

    if (tid == 0) {
        for (int s = 0; s < G::NSTAGE; s++) {
            mbar_init(&bar[s], 1);
            mbar_init(&face_bar[s], (uint32_t)NT);
        }
        mbar_init(psi_bar, (uint32_t)(NT / 32));
        *s_fail = 0;
        mbar_init_fence();
    }
    __syncthreads();

    auto box_ptr = [&](int s, int b) -> double* {
        return reinterpret_cast<double*>(stage0 + s * G::STAGE_BYTES + b * G::BOX_PITCH);
    };
    // Request plane p (z0-1 <= p <= z1) into stage s.
    auto fill = [&](int p, int s) {
        if (tid != 0) return;
        mbar_arrive_expect_tx(&bar[s], (uint32_t)(G::NBOX * G::BOX_BYTES));
        static_for<15>([&](auto kk) {
            constexpr int k = decltype(kk)::value;
            tma_load_4d(box_ptr(s, k), &tm_f, x0 - 2, y0 - 1 - cyk<L>(k), wrap_any(p - czk<L>(k), nz), k, &bar[s]);
        });
        tma_load_3d(box_ptr(s, 15), &tm_T, x0 - 2, y0 - 1, wrap_any(p, nz), &bar[s]);
    };
    // Face tiles: the wrapped parts of plane p, once its tensor copies have landed.
    auto patch = [&](int p, int s) {
        auto cy = [](int b) { return b < 15 ? cyk<L>(b) : 0; };
        patch_wrapped<TX, TY, G::NBOX>(tid, NT, x0, y0, nx, ny, cy,
                                       [&](int b, int iy, int y, unsigned char*& dst, const unsigned char*& src, int& es) {
            const int z = wrap_any(p - (b < 15 ? czk<L>(b) : 0), nz);
            es = 8;
            dst = (unsigned char*)(box_ptr(s, b) + iy * G::BX);
            src = (const unsigned char*)((b < 15 ? A.fin + (size_t)b * n : A.Told) + (size_t)nx * ((size_t)y + (size_t)ny * z));
        }, [](unsigned char* dst, const unsigned char* src) { cp_async16(dst, src); },
           [&](unsigned char* dst, const unsigned char* src, int bytes) {
               mbar_expect_tx(&face_bar[s], (uint32_t)bytes);
               bulk_load(dst, src, (uint32_t)bytes, &face_bar[s]);
           });
    };

    // per stage, bit s: the parity of its next waits, and whether tensor copies are outstanding
    uint32_t parity = 0, fparity = 0, pending = 0;
    auto arrived = [&](int s) {  // the tensor copies of stage s have landed
        const bool ok = mbar_wait_bounded(&bar[s], (parity >> s) & 1u, TMA_WAIT_LIMIT);
        if (ok) {
            parity ^= 1u << s;
            pending &= ~(1u << s);
        }
        return ok;
    };
    const int pfirst = z0 - 1, plast = z1;  // psi is needed on planes z0-1 .. z1
    for (int q = 0; q < G::NSTAGE && pfirst + q <= plast; q++) {
        fill(pfirst + q, q);
        pending |= 1u << q;
    }
    if (face) {
        if (arrived(0)) patch(pfirst, 0);
        else *s_fail = 1;
        mbar_arrive_cp_async(&face_bar[0]);
    }

    double fp[15] = {}, fc[15];  // own pulled populations: plane p-1 (collided now), plane p (next)
    double rp = 0, rrp = 0, rc = 0, rrc = 0;
    bool failed = false;
    for (int p = pfirst; p <= plast; p++) {
        const int j = p - pfirst, s = j % G::NSTAGE;
        const bool landed = face ? mbar_wait_bounded(&face_bar[s], (fparity >> s) & 1u, TMA_WAIT_LIMIT) : arrived(s);
        fparity ^= 1u << s;
        // psi of plane p: ring slots, then the own slot (whose populations
        // stay in registers).  Population k of ext slot (ex, ey) sits at
        // box k, row ey, column ex + 1 - c_kx; T at box 15, column ex + 1.
        const double* sb = box_ptr(s, 0);
        constexpr int BP = G::BOX_PITCH / 8;
        double(*psi_p)[EX] = s_psi[(p + G::NPSI) % G::NPSI];
        for (int r = tid; landed && r < NRING; r += NT) {
            int ex, ey;
            ring_slot(r, TX, TY, ex, ey);
            const double* sl = sb + ey * G::BX + ex + 1;
            double rho = 0;
            static_for<15>([&](auto kk) {
                constexpr int k = decltype(kk)::value;
                rho += sl[k * BP - cxk<L>(k)];
            });
            psi_p[ey][ex] = potential(P, rho, sl[15 * BP]);
        }
        if (landed) {
            const int ex = tx + 1, ey = ty + 1;
            const double* sl = sb + ey * G::BX + ex + 1;
            double rho = 0;
            static_for<15>([&](auto kk) {
                constexpr int k = decltype(kk)::value;
                fc[k] = sl[k * BP - cxk<L>(k)];
                rho += fc[k];
            });
            rc = rho;
            rrc = rcp_rn(rho);
            psi_p[ey][ex] = potential(P, rho, sl[15 * BP]);
        }
        // arrive: this warp's psi of plane p is written and its stage read
        if (!landed) *s_fail = 1;
        if (face) fence_proxy_async_smem();  // the stage's next tensor copy follows the writes of patch()
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(psi_bar);
        double m[15];  // moments of plane p-1 (moment 0 is rho)
        mul_M<L, 1>(fp, m);
        // one decision for the whole block: a wait that ran out in any thread ends the kernel
        if (!mbar_wait_bounded(psi_bar, (uint32_t)j & 1u, TMA_WAIT_LIMIT) || *s_fail) {
            *s_fail = 1;
            if (face)
                leave_face_tile(j, G::NSTAGE, fparity, p + 1 <= plast, [&](int t) { mbar_arrive(&face_bar[t]); },
                                [&](int t, uint32_t par) { mbar_wait_bounded(&face_bar[t], par, TMA_WAIT_LIMIT); });
            failed = true;
            break;
        }
        // stage s has been read: request plane p + NSTAGE into it
        if (p + G::NSTAGE <= plast) {
            fill(p + G::NSTAGE, s);
            pending |= 1u << s;
        }
        // plane p + 1, requested one plane ago: write its wrapped parts
        if (face && p + 1 <= plast) {
            const int t = (j + 1) % G::NSTAGE;
            if (arrived(t)) patch(p + 1, t);
            else *s_fail = 1;
            mbar_arrive_cp_async(&face_bar[t]);
        }
        // collide plane p-1 with psi of planes p-2, p-1, p
        const int z = p - 1;
        if (z >= z0) {
            const uint32_t id = (uint32_t)(x0 + tx) + (uint32_t)nx * ((uint32_t)(y0 + ty) + (uint32_t)ny * (uint32_t)z);
            const int ex = tx + 1, ey = ty + 1;
            auto nbpsi = [&](int k) {
                return s_psi[(z + czk<L>(k) + G::NPSI) % G::NPSI][ey + cyk<L>(k)][ex + cxk<L>(k)];
            };
            finish_moments<ST>(P, A, id, m, rp, rrp, s_psi[(z + G::NPSI) % G::NPSI][ey][ex], nbpsi);
        }
#pragma unroll
        for (int k = 0; k < 15; k++) fp[k] = fc[k];
        rp = rc;
        rrp = rrc;
    }
    if (failed) {
        if (tid == 0) atomicExch(A.kerr, MPLB_KERR_WAIT);
        // let the copies this block issued land before its shared memory is released
        // (the bulk copies of wrapped parts: leave_face_tile)
        cp_async_wait_all();
        for (int s = 0; s < G::NSTAGE; s++)
            if ((pending >> s) & 1u) mbar_wait_bounded(&bar[s], (parity >> s) & 1u, TMA_WAIT_LIMIT);
    }
}

// Fully periodic D3Q15 box without boundary programs, tiles that divide
// the box, an even x extent: the lattices this kernel takes.
inline bool tma3_fits(const FusedArgs& A, bool has_bc, int TX, int TY) {
    return !has_bc && A.px && A.py && A.pz && A.nx % TX == 0 && A.ny % TY == 0 && A.nx % 2 == 0 && A.nz >= 2;
}

}  // namespace mplb
