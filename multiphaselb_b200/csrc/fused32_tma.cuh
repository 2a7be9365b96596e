// fused32_tma.cuh -- the FP32-deviation D3Q15 step with the plane neighbourhood
// staged by TMA: the scheme of fused_tma.cuh (fully periodic boxes without
// boundary programs; one tensor copy per population and plane, the wrapped
// parts of face tiles written after it; two plane stages, four psi planes, one
// split barrier per plane) on FP32 populations.
//
// For population k the tile's pull sources on plane z - c_kz are one box of
// (TX+8) x (TY+2) floats from (x0-4, y0-1-c_ky): x0-4 is a multiple of four,
// so the box starts on a 16-byte boundary.  T stays FP64, in a box of its own.
//
// Bound by issue and latency (FP64 force and EOS, about 55 conversions between
// FP32 and FP64 a node) at one 512-thread block per SM.  B200, 192^3: 338 us a
// step; the general kernel, which computes 1.8 psi per node and loads each
// population with its own address, takes 438.
#pragma once

#include "fused32.cuh"
#include "tma_maps.h"
#include "tma_util.cuh"

namespace mplb {

template <int TX, int TY>
struct TmaTile32 {
    static constexpr int BX = TX + 8, BY = TY + 2;   // population boxes, floats, x from x0-4
    static constexpr int TBX = TX + 4;               // T box, doubles, x from x0-2
    static constexpr int BOX_BYTES = BX * BY * 4, T_BYTES = TBX * BY * 8;
    static constexpr int BOX_PITCH = (BOX_BYTES + 127) / 128 * 128, T_PITCH = (T_BYTES + 127) / 128 * 128;
    static constexpr int STAGE_BYTES = 15 * BOX_PITCH + T_PITCH;
    static constexpr int NSTAGE = 2, NPSI = 4, HEAD = 128;
    static constexpr int EX = TX + 2, EY = TY + 2;
    static constexpr size_t SMEM = 128 + HEAD + (size_t)NSTAGE * STAGE_BYTES + (size_t)NPSI * EY * EX * 8;
    static_assert(TX % 4 == 0, "x0 - 4 must be a multiple of four");
};

// Candidate box: what the kernel takes.
inline bool tma3_fits32(int nx, int ny, int nz, int px, int py, int pz, bool has_bc, int TX, int TY) {
    return !has_bc && px && py && pz && nx % TX == 0 && ny % TY == 0 && nz >= 2;
}

// The kernel that steps a box without boundary programs: 0, 1 the TMA-staged one
// with 64 x 8 tiles (one block per SM) or 32 x 8 (two, more halo per node), -1
// the general one.  By an estimate of its time, in us on a B200: rounds of
// resident blocks, times the planes of a block, times what a plane took.  The
// TMA kernel's plane is the longer one: 3.5 us; with 32 x 8 tiles 2.8, two per
// SM 3.6; a fifth more where a tile's rows lie on both y faces; general 2.25,
// 2.75, 3.25 and 3.95 with one to four blocks per SM, 5.5 with five.  Its chunks
// may be shorter, though, four planes instead of eight, to fill the device.
// (The planes beside a chunk count in full but for the general kernel at four
// and more blocks per SM, and a round that is not full costs that kernel half of
// one, unless nearly empty.)  So flat boxes and slabs of a few planes take the
// general kernel and large boxes the TMA one.  Measured, us per step, general,
// 64 x 8, 32 x 8: 64 x 8 x 4 13.8, 24.7, 21.2; 64 x 64 x 4 14.0, 21.9, 18.1;
// 320 x 320 x 2 18.9, 28.6, 25.1; 512 x 512 x 2 46.6, 55.4, 50.1; 64 x 64 x 16
// 24.5, 22.3, 18.3; 192 x 192 x 8 28.7, 23.6, 24.0; 512 x 512 x 16 250, 252, 242;
// 128^3 126, 121, 127; 192^3 438, 338, 357.
inline int tma32_tile(const FusedArgs& A, bool has_bc) {
    if (!tma3_fits32(A.nx, A.ny, A.nz, A.px, A.py, A.pz, has_bc, 32, 8)) return -1;
    const double edge = A.ny == 8 ? 1.2 : 1.0;
    const Geom g = fused_geometry(MPLB_D3Q15, A, 32, 4);
    const double per_sm = g.nblocks / 148.0;
    const double rounds = (double)g.tiles_x * g.tiles_y * A.nz / g.zchunk / (5 * 148);
    double best = general32_blocks(g, A.nz) == 4 ? (g.zchunk + 1.6) * 3.95
                  : per_sm <= 4 ? (g.zchunk + 2) * (per_sm <= 1 ? 2.25 : per_sm <= 2 ? 2.75 : 3.25)
                                : (g.zchunk + 1.3) * 5.5 * (rounds <= 1.2 ? std::max(1.0, rounds) : std::max(1.5, rounds));
    int pick = -1;
    if (A.nx % 64 == 0) {
        const Geom t = resident_geometry(A, 64, 8, 1);
        const double us = 1.2 + (t.zchunk + 2) * edge * 3.5 * ((t.nblocks + 147) / 148);
        if (us < best) {
            best = us;
            pick = 0;
        }
    }
    const Geom t = resident_geometry(A, 32, 8, 2);
    const int rest = t.nblocks % 296;
    const double us = 1.2 + (t.zchunk + 2) * edge * (3.6 * (t.nblocks / 296) + (rest == 0 ? 0.0 : rest <= 148 ? 2.8 : 3.6));
    return us < best ? 1 : pick;
}

// That kernel and, for the TMA-staged one, the tensor maps of the step's input
// buffers.  tile -1: the general kernel (the box, or no maps to be had).
struct Tma32 {
    int tile = -1;  // 0: 64 x 8, 1: 32 x 8
    const TmaMaps* maps = nullptr;
};
inline Tma32 tma32_choose(TmaMapCache& cache, PFN_cuTensorMapEncodeTiled_v12000 enc, const FusedArgs& A, bool has_bc,
                          uint32_t n, const float* fin, const double* Told) {
    Tma32 r;
    r.tile = tma32_tile(A, has_bc);
    if (r.tile < 0) return r;
    const int tx = r.tile == 0 ? 64 : 32, ty = 8;
    r.maps = cache.get(enc, r.tile, A.nx, A.ny, A.nz, fin, true, Told, n, tx + 8, ty + 2, tx + 4);
    if (!r.maps) r.tile = -1;
    return r;
}

template <int TX, int TY, int MINB>
__global__ void __launch_bounds__(TX * TY, MINB)
    k_fused32_d3q15_tma(Params P, FusedArgs32 A, const __grid_constant__ CUtensorMap tm_f,
                        const __grid_constant__ CUtensorMap tm_T) {
    step_dependency_wait();
    using L = D3Q15T;
    using G = TmaTile32<TX, TY>;
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
    const uint32_t n = A.n;
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

    auto box = [&](int s, int k) { return reinterpret_cast<float*>(stage0 + s * G::STAGE_BYTES + k * G::BOX_PITCH); };
    auto tbox = [&](int s) { return reinterpret_cast<double*>(stage0 + s * G::STAGE_BYTES + 15 * G::BOX_PITCH); };
    // Request plane p (z0-1 <= p <= z1) into stage s.
    auto fill = [&](int p, int s) {
        if (tid != 0) return;
        mbar_arrive_expect_tx(&bar[s], (uint32_t)(15 * G::BOX_BYTES + G::T_BYTES));
        static_for<15>([&](auto kk) {
            constexpr int k = decltype(kk)::value;
            tma_load_4d(box(s, k), &tm_f, x0 - 4, y0 - 1 - cyk<L>(k), wrap_any(p - czk<L>(k), nz), k, &bar[s]);
        });
        tma_load_3d(tbox(s), &tm_T, x0 - 2, y0 - 1, wrap_any(p, nz), &bar[s]);
    };
    // Face tiles: the wrapped parts of plane p, once its tensor copies have landed.
    auto patch = [&](int p, int s) {
        auto cy = [](int b) { return b < 15 ? cyk<L>(b) : 0; };
        patch_wrapped<TX, TY, 16>(tid, NT, x0, y0, nx, ny, cy,
                                  [&](int b, int iy, int y, unsigned char*& dst, const unsigned char*& src, int& es) {
            const bool pop = b < 15;
            const size_t row = (size_t)nx * ((size_t)y + (size_t)ny * wrap_any(p - (pop ? czk<L>(b) : 0), nz));
            es = pop ? 4 : 8;
            dst = pop ? (unsigned char*)(box(s, b) + iy * G::BX) : (unsigned char*)(tbox(s) + iy * G::TBX);
            src = pop ? (const unsigned char*)(A.fin + (size_t)b * n + row) : (const unsigned char*)(A.Told + row);
        }, [](unsigned char* dst, const unsigned char* src) { cp_async16(dst, src); },
           [&](unsigned char* dst, const unsigned char* src, int bytes) {
               mbar_expect_tx(&face_bar[s], (uint32_t)bytes);
               bulk_load(dst, src, (uint32_t)bytes, &face_bar[s]);
           });
    };

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

    float fp[15] = {}, fc[15];  // own pulled deviations: plane p-1 (collided now), plane p (next)
    double rp = 0, rc = 0;
    float drp = 0.f, drc = 0.f;
    bool failed = false;
    for (int p = pfirst; p <= plast; p++) {
        const int j = p - pfirst, s = j % G::NSTAGE;
        const bool landed = face ? mbar_wait_bounded(&face_bar[s], (fparity >> s) & 1u, TMA_WAIT_LIMIT) : arrived(s);
        fparity ^= 1u << s;
        // psi of plane p: population k of ext slot (ex, ey) sits at box k, row
        // ey, column ex + 3 - c_kx; T at column ex + 1 of its box
        const float* sb = box(s, 0);
        const double* st = tbox(s);
        constexpr int BP = G::BOX_PITCH / 4;
        double(*psi_p)[EX] = s_psi[(p + G::NPSI) % G::NPSI];
        for (int r = tid; landed && r < NRING; r += NT) {
            int ex, ey;
            ring_slot(r, TX, TY, ex, ey);
            const float* sl = sb + ey * G::BX + ex + 3;
            float d = 0.f;
            static_for<15>([&](auto kk) {
                constexpr int k = decltype(kk)::value;
                d += sl[k * BP - cxk<L>(k)];
            });
            psi_p[ey][ex] = potential(P, A.rho_ref + (double)d, st[ey * G::TBX + ex + 1]);
        }
        if (landed) {
            const int ex = tx + 1, ey = ty + 1;
            const float* sl = sb + ey * G::BX + ex + 3;
            float d = 0.f;
            static_for<15>([&](auto kk) {
                constexpr int k = decltype(kk)::value;
                fc[k] = sl[k * BP - cxk<L>(k)];
                d += fc[k];
            });
            drc = d;
            rc = A.rho_ref + (double)d;
            psi_p[ey][ex] = potential(P, rc, st[ey * G::TBX + ex + 1]);
        }
        // arrive: this warp's psi of plane p is written and its stage read
        if (!landed) *s_fail = 1;
        if (face) fence_proxy_async_smem();  // the stage's next tensor copy follows the writes of patch()
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(psi_bar);
        Pre32<L> q;
        pre_node32<L>(fp, q);  // plane p-1: what needs no neighbour
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
            const double psi = s_psi[(z + G::NPSI) % G::NPSI][ey][ex];
            double Fi[3], Ft[3], Ud[3];
            force_velocity32<L>(P, false, q.m, rp, psi, nbpsi, Fi, Ft, Ud);
            float f[15];
            collide_node32<L>(P, A, q, f, rp, drp, psi, Fi, Ft, Ud);
#pragma unroll
            for (int k = 0; k < 15; k++) A.fout[(size_t)k * n + id] = f[k];
        }
#pragma unroll
        for (int k = 0; k < 15; k++) fp[k] = fc[k];
        rp = rc;
        drp = drc;
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

}  // namespace mplb
