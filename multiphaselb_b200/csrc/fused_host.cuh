// fused_host.cuh -- host side of the fused box path: boundary-program
// tables, candidate launches, the tile autotuner.  Included only by the FP64
// translation unit, so the FP64 kernels are instantiated in exactly one
// object (compiled without multiply-add contraction).
#pragma once

#include "fused.cuh"
#include "fused_launch.cuh"
#include "fused_march.cuh"
#include "fused_table.cuh"
#include "fused_tma.cuh"
#include "tma_maps.h"

// The marching D2Q9 step with myMRT heat (mplb_march.cu).
int mplb_march_resident(bool f_on, bool bc);
cudaError_t mplb_march_launch(bool f_on, bool bc, int nb, const mplb::Params& P, const mplb::FusedArgs& A, cudaStream_t s);

// The general steps with a surface-tension term (mplb_st.cu).
cudaError_t mplb_st_attributes();
void mplb_st_launch2(int cfg, bool g_on, bool bc, int nb, const mplb::Params& P, const mplb::FusedArgs& A, cudaStream_t s);
void mplb_st_launch3(int cfg, bool bc, int nb, const mplb::Params& P, const mplb::FusedArgs& A, cudaStream_t s);

// Steps on neighbour tables (mplb_table.cu); returns the launches made.
int mplb_table_step(int lat, int heat, bool emit, bool st, const mplb::Params& P, const mplb::TableArgs& A,
                    cudaStream_t s);

namespace mplb {

// While this lives, the calling thread may allocate and wait although some other
// stream is being captured (a step of this handle is no part of that capture,
// and the operators, which the table kernels stand for, allocate nothing).
struct AnyCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    AnyCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~AnyCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

struct FusedConfig {
    std::string err;
    FusedArgs args{};
    uint8_t* bcmap = nullptr;
    bool has_bc = false;
    int lat = 0;
    int cfg = 0;           // chosen candidate
    bool tuned = false;    // autotuner has run (or a candidate was forced)
    Geom geom[N_CFG_MAX];
    float tune_ms[N_CFG_MAX] = {};
    int ncfg = 0;
    int nblocks = 0;
    double* my_scratch = nullptr;  // myMRT: rho_a and gsum_a, 2 n doubles
    // table candidate (D3Q15): table, flags and scratch (table_scratch); the best
    // tile candidate, which takes the steps of slabs (owned and mirrored ranges)
    TableArgs tab{};
    int tile_cfg = 2;
    int* kerr = nullptr;           // kernel error flag (bounded waits), one int
    int* kerr_host = nullptr;      // its pinned host copy
    TmaMapCache tmaps;
};

// The 3D kernels use more than the 48 KB of static shared memory.
inline cudaError_t fused_attributes() {
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    chk(set_smem3<32, 8, false, true, true>());
    chk(set_smem3<32, 8, false, false, true>());
    chk(general_attributes<false>());
    chk(mplb_st_attributes());
#define MPLB_SET3_TMA(TX, TY, MINB)                                                                                          \
    chk(cudaFuncSetAttribute(k_fused_d3q15_tma<TX, TY, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,                  \
                             (int)TmaTile<TX, TY>::SMEM));                                                                  \
    chk(cudaFuncSetAttribute(k_fused_d3q15_tma<TX, TY, MINB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,            \
                             (int)TmaTile<TX, TY>::SMEM));
    MPLB_SET3_TMA(32, 4, 3)
    MPLB_SET3_TMA(32, 8, 2)
    MPLB_SET3_TMA(32, 16, 1)
    MPLB_SET3_TMA(64, 8, 1)
#undef MPLB_SET3_TMA
    return e;
}

template <int TX, int TY, int MINB>
cudaError_t launch3_tma(FusedConfig& fc, int cfg, int nb, const Params& P, const FusedArgs& A, cudaStream_t s) {
    const TmaMaps* m = fc.tmaps.get(tensor_map_encoder(), cfg, A.nx, A.ny, A.nz, A.fin, false, A.Told, P.n, TX + 4, TY + 2,
                                    TX + 4);
    if (!m) return cudaErrorInvalidValue;
    if (P.st_on) launch_step(k_fused_d3q15_tma<TX, TY, MINB, true>, nb, TX * TY, TmaTile<TX, TY>::SMEM, s, P, A, m->mf, m->mT);
    else launch_step(k_fused_d3q15_tma<TX, TY, MINB>, nb, TX * TY, TmaTile<TX, TY>::SMEM, s, P, A, m->mf, m->mT);
    return cudaSuccess;
}

// myMRT steps first fill rho_a, gsum_a (k_pullsum_d2q9).
template <bool F_ON>
void launch_pullsum(bool bc, const Params& P, const FusedArgs& A, cudaStream_t s) {
    const unsigned nb = (P.n + 255) / 256;
    if (bc) launch_step(k_pullsum_d2q9<F_ON, true>, nb, 256, 0, s, P, A);
    else launch_step(k_pullsum_d2q9<F_ON, false>, nb, 256, 0, s, P, A);
}

// The table candidate takes steps that store every node; the others run on the
// best tile candidate (fc.tile_cfg), as all do without its scratch.
inline bool table_whole(const Params& P, const FusedArgs& A) { return A.own_cnt == P.n && !A.nmirror; }

// That scratch, a double a node: had when the tuner keeps the candidate or a
// caller forces it.
inline void table_scratch(FusedConfig& fc, uint32_t n, uint64_t* bytes) {
    if (fc.tab.psi) return;
    AnyCapture guard;
    if (cudaMalloc((void**)&fc.tab.psi, (size_t)n * sizeof(double)) == cudaSuccess) {
        *bytes += (size_t)n * sizeof(double);
    } else {
        cudaGetLastError();
        fc.tab.psi = nullptr;
    }
}
inline void table_scratch_free(FusedConfig& fc, uint32_t n, uint64_t* bytes) {
    if (!fc.tab.psi) return;
    cudaFree(fc.tab.psi);
    fc.tab.psi = nullptr;
    *bytes -= (size_t)n * sizeof(double);
}

// Launch one fused step with candidate `cfg` (EMIT always uses candidate 0);
// *launches: the kernels that takes.
inline cudaError_t fused_launch_cfg(FusedConfig& fc, int cfg, const Params& P, FusedArgs A, bool f_on, bool g_on,
                                    bool emit, cudaStream_t s, int* launches) {
    *launches = 1;
    if (fc.lat == MPLB_D3Q15 && CFG3[cfg].table && !emit) {
        if (fc.tab.psi && table_whole(P, A)) {
            TableArgs T = fc.tab;
            T.fin = A.fin;
            T.fout = A.fout;
            T.Told = A.Told;
            T.Uold = A.Uold;
            T.Unew = A.Unew;
            T.rho = A.rho_out;  // rewritten with the reference state
            *launches = mplb_table_step(fc.lat, TABLE_NONE, false, P.st_on != 0, P, T, s);
            return cudaGetLastError();
        }
        cfg = fc.tile_cfg;
    }
    if (fc.geom[cfg].nblocks == 0 && !emit) return cudaErrorInvalidConfiguration;  // the candidate does not take this lattice
    if (emit) cfg = 0;
    apply_geom(A, fc.geom[cfg]);
    const int nb = fc.geom[cfg].nblocks;
    const bool bc = fc.has_bc, st = P.st_on && f_on;
    if (fc.lat == MPLB_D2Q9) {
        if (emit) {
            launch2_fg<32, 8, true>(f_on, g_on, bc, nb, P, A, s);
        } else if (CFG2[cfg].march) {
            return mplb_march_launch(f_on, bc, nb, P, A, s);
        } else {
            if (g_on && P.g_model == MPLB_MYMRT) {
                *launches = 2;
                if (f_on) launch_pullsum<true>(bc, P, A, s);
                else launch_pullsum<false>(bc, P, A, s);
            }
            if (st) mplb_st_launch2(cfg, g_on, bc, nb, P, A, s);
            else launch_general2<false>(cfg, f_on, g_on, bc, nb, P, A, s);
        }
    } else {
        if (emit) {
            launch3<32, 8, false, true>(bc, nb, P, A, s);
        } else if (!CFG3[cfg].tma) {
            if (st) mplb_st_launch3(cfg, bc, nb, P, A, s);
            else launch_general3<false>(cfg, bc, nb, P, A, s);
        } else {
            switch (cfg) {
            case 6: if (cudaError_t e = launch3_tma<32, 4, 3>(fc, cfg, nb, P, A, s)) return e; break;
            case 7: if (cudaError_t e = launch3_tma<32, 8, 2>(fc, cfg, nb, P, A, s)) return e; break;
            case 8: if (cudaError_t e = launch3_tma<32, 16, 1>(fc, cfg, nb, P, A, s)) return e; break;
            default: if (cudaError_t e = launch3_tma<64, 8, 1>(fc, cfg, nb, P, A, s)) return e; break;
            }
        }
    }
    return cudaGetLastError();
}

inline cudaError_t fused_launch(FusedConfig& fc, const Params& P, const FusedArgs& A, bool f_on, bool g_on, bool emit,
                                cudaStream_t s, int* launches) {
    return fused_launch_cfg(fc, fc.cfg, P, A, f_on, g_on, emit, s, launches);
}

// Time every candidate on the current state and keep the fastest.  Three
// sweeps over the candidates (so a transient -- clocks settling, another
// process -- does not favour the candidates timed during it); in each, a
// candidate's warm-up launch and 8 timed launches are queued back to back
// with an event between consecutive launches and one host wait at the end,
// so a launch's interval holds its device time only (a host wait between
// launches would add the host's launch latency, several microseconds, to
// every interval: on a lattice of one wave that is as large as the
// differences between candidates).  A candidate's time is the median of its
// 24 intervals.  The step's outputs are rewritten by the real launch that
// follows; the heat-source history S, updated in place, is saved to `save`
// before and restored after every candidate's launches.
inline int fused_autotune(FusedConfig& fc, const Params& P, const FusedArgs& A, bool f_on, bool g_on, double* S,
                          double* save, size_t n, cudaStream_t s, uint64_t* bytes) {
    constexpr int SWEEPS = 3, WARM = 1, TIMED = 8;
    cudaEvent_t ev[TIMED + 1];
    int made = 0;
    for (; made < TIMED + 1; made++)
        if (cudaEventCreate(&ev[made]) != cudaSuccess) break;
    if (made < TIMED + 1) {
        for (int i = 0; i < made; i++) cudaEventDestroy(ev[i]);
        fc.err = "autotune: event creation failed";
        return MPLB_E_CUDA;
    }
    const bool keep_s = g_on && S && save;
    if (keep_s && cudaMemcpyAsync(save, S, n * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
        for (int i = 0; i < TIMED + 1; i++) cudaEventDestroy(ev[i]);
        fc.err = "autotune: saving S failed";
        return MPLB_E_CUDA;
    }
    float ms_all[N_CFG_MAX][SWEEPS * TIMED];
    bool ok_c[N_CFG_MAX];
    // the table candidate is timed on `save`, which these lattices do not need:
    // an allocation that another candidate's win would undo takes 0.5 to 1 ms
    const bool lent = fc.lat == MPLB_D3Q15 && table_whole(P, A) && !fc.tab.psi && !keep_s;
    if (lent) fc.tab.psi = save;
    for (int c = 0; c < fc.ncfg; c++) {
        ok_c[c] = fc.geom[c].nblocks > 0;
        if (fc.lat == MPLB_D3Q15 && CFG3[c].table) ok_c[c] = fc.tab.psi && table_whole(P, A);
    }
    for (int sw = 0; sw < SWEEPS; sw++) {
        for (int c = 0; c < fc.ncfg; c++) {
            bool ok = ok_c[c];
            for (int r = 0; r < WARM + TIMED && ok; r++) {
                if (r >= WARM) cudaEventRecord(ev[r - WARM], s);
                int launches;
                ok = fused_launch_cfg(fc, c, P, A, f_on, g_on, false, s, &launches) == cudaSuccess;
            }
            if (ok) cudaEventRecord(ev[TIMED], s);
            if (ok && cudaEventSynchronize(ev[TIMED]) == cudaSuccess) {
                for (int r = 0; r < TIMED; r++) {
                    float ms = 0;
                    cudaEventElapsedTime(&ms, ev[r], ev[r + 1]);
                    ms_all[c][sw * TIMED + r] = ms;
                }
            } else {
                ok = false;
            }
            if (keep_s) cudaMemcpyAsync(S, save, n * sizeof(double), cudaMemcpyDeviceToDevice, s);
            ok_c[c] = ok;
        }
    }
    float best = 1e30f;
    int best_cfg = 0;
    for (int c = 0; c < fc.ncfg; c++) {
        float med = -1.0f;
        if (ok_c[c]) {
            float* m = ms_all[c];
            std::sort(m, m + SWEEPS * TIMED);
            med = 0.5f * (m[SWEEPS * TIMED / 2 - 1] + m[SWEEPS * TIMED / 2]);
        }
        fc.tune_ms[c] = ok_c[c] ? med : -1.0f;
        if (ok_c[c] && med >= 0 && med < best) {
            best = med;
            best_cfg = c;
        }
    }
    if (fc.lat == MPLB_D3Q15) {
        best = 1e30f;
        for (int c = 0; c < fc.ncfg; c++)
            if (!CFG3[c].table && ok_c[c] && fc.tune_ms[c] < best) {
                best = fc.tune_ms[c];
                fc.tile_cfg = c;
            }
    }
    cudaGetLastError();
    for (int i = 0; i < TIMED + 1; i++) cudaEventDestroy(ev[i]);
    if (lent) {
        fc.tab.psi = nullptr;
        if (CFG3[best_cfg].table) table_scratch(fc, P.n, bytes);
        if (CFG3[best_cfg].table && !fc.tab.psi) best_cfg = fc.tile_cfg;
    }
    fc.cfg = best_cfg;
    fc.nblocks = fc.geom[best_cfg].nblocks;
    fc.tuned = true;
    return cudaStreamSynchronize(s) == cudaSuccess ? 0 : MPLB_E_CUDA;
}

// Fused path preconditions: box mesh, no serial boundary dependence, only
// bounceBack / fixedT / periodic patches, at most FUSED_MAX_OPS ops per node
// and field, at most FUSED_MAX_PROGS distinct node programs.
inline bool fused_supported(int lat, const int* model, const Params& P, const std::vector<PatchDev>* fp,
                            const bool* serial, const mplb_mesh_desc* mesh, const int* dims, const int* per,
                            std::string& why) {
    (void)per;
    const bool active[2] = {model[0] != MPLB_NO_MODEL && P.f_update != 0, model[1] != MPLB_NO_MODEL && P.g_update != 0};
    if (serial[0] || serial[1]) { why = "boundary updates depend on the serial order"; return false; }
    if (!active[0] && !active[1]) { why = "no field is updated"; return false; }
    if (!active[0] && model[0] == MPLB_NO_MODEL) { why = "no flow field"; return false; }
    if (lat == MPLB_D3Q15 && active[1]) { why = "thermal field on D3Q15"; return false; }
    for (int fi = 0; fi < 2; fi++) {
        if (!active[fi]) continue;
        for (const PatchDev& pt : fp[fi]) {
            if (pt.type == MPLB_BC_PERIODIC) continue;
            if (pt.type == MPLB_BC_BOUNCEBACK) continue;
            if (pt.type == MPLB_BC_FIXEDT && fi == 1) continue;
            if (pt.type == MPLB_BC_FIXEDU && model[fi] != MPLB_LIMRT) continue;  // no-op
            why = "boundary type " + std::to_string(pt.type) + " is handled by the operator path only";
            return false;
        }
    }
    if (dims[0] < 2 || dims[1] < 2 || (lat == MPLB_D3Q15 && dims[2] < 2)) { why = "box thinner than 2 nodes"; return false; }
    (void)mesh;
    return true;
}

// The boundary program of every node (index into progs; 0 = none).
inline int node_programs(const Params& P, const std::vector<PatchDev>* fp, const mplb_mesh_desc* mesh,
                         std::vector<uint8_t>& map, std::vector<BCProg>& progs, bool& any, std::string& err) {
    // Node programs: for every node, the ops of every patch holding it, in
    // patch order, per field.  Identical programs share one table entry.
    const uint32_t n = P.n;
    map.assign(n, 0);
    progs.assign(1, BCProg{});
    any = false;
    {
        // programs of the patches' nodes only: an entry for every node of a large
        // lattice would cost its page faults at each create
        std::vector<uint32_t> slot(n, 0);
        std::vector<BCProg> node(1, BCProg{});
        size_t off = 0;
        for (size_t p = 0; p < fp[0].size(); p++) {
            for (uint32_t i = 0; i < fp[0][p].count; i++) {
                uint32_t id = mesh->patch_nodes[off + i];
                for (int fi = 0; fi < 2; fi++) {
                    if (!(fi == 0 ? P.f_update : P.g_update)) continue;
                    int t = fp[fi][p].type;
                    if (t != MPLB_BC_BOUNCEBACK && t != MPLB_BC_FIXEDT) continue;
                    if (!slot[id]) {
                        slot[id] = (uint32_t)node.size();
                        node.push_back(BCProg{});
                    }
                    BCProg& b = node[slot[id]];
                    if (fi == 0) {
                        if (b.nf >= FUSED_MAX_OPS) { err = "too many boundary ops on one node"; return MPLB_E_UNSUPPORTED; }
                        b.ft[b.nf++] = (uint8_t)t;
                    } else {
                        if (b.ng >= FUSED_MAX_OPS) { err = "too many boundary ops on one node"; return MPLB_E_UNSUPPORTED; }
                        b.gp[b.ng] = (uint8_t)p;
                        b.gt[b.ng++] = (uint8_t)t;
                    }
                    any = true;
                }
            }
            off += fp[0][p].count;
        }
        for (uint32_t id = 0; id < n; id++) {
            if (!slot[id]) continue;
            const BCProg& b = node[slot[id]];
            int found = -1;
            for (size_t q = 1; q < progs.size(); q++)
                if (std::memcmp(&progs[q], &b, sizeof(BCProg)) == 0) { found = (int)q; break; }
            if (found < 0) {
                if (progs.size() >= FUSED_MAX_PROGS) { err = "too many distinct boundary programs"; return MPLB_E_UNSUPPORTED; }
                progs.push_back(b);
                found = (int)progs.size() - 1;
            }
            map[id] = (uint8_t)found;
        }
    }
    return 0;
}

inline int fused_setup(FusedConfig& fc, int lat, const int* model, const Params& P, const std::vector<PatchDev>* fp,
                       const mplb_mesh_desc* mesh, const int* dims, const int* per, const int32_t* nb,
                       const uint8_t* onb, cudaStream_t stream, uint64_t* bytes) {
    FusedArgs& A = fc.args;
    A.nx = dims[0];
    A.ny = dims[1];
    A.nz = lat == MPLB_D3Q15 ? dims[2] : 1;
    A.px = per[0];
    A.py = per[1];
    A.pz = lat == MPLB_D3Q15 ? per[2] : 1;
    A.own_lo = 0;
    A.own_cnt = P.n;  // every node's outputs stored; slabs narrow it (mplb_gpu_set_owned)
    A.nmirror = 0;
    std::vector<uint8_t> map;
    std::vector<BCProg> progs;
    bool any = false;
    if (int rc = node_programs(P, fp, mesh, map, progs, any, fc.err)) return rc;
    const uint32_t n = P.n;
    // farthest distance of a node with a boundary program from its nearest
    // box face (-1: none); tiles whose ring lies farther in hold none
    A.bc_margin = -1;
    for (uint32_t id = 0; id < n; id++) {
        if (!map[id]) continue;
        const int x = (int)(id % (uint32_t)A.nx), y = (int)((id / (uint32_t)A.nx) % (uint32_t)A.ny);
        const int z = (int)(id / ((uint32_t)A.nx * (uint32_t)A.ny));
        int d = std::min(std::min(x, A.nx - 1 - x), std::min(y, A.ny - 1 - y));
        if (lat == MPLB_D3Q15) d = std::min(d, std::min(z, A.nz - 1 - z));
        A.bc_margin = std::max(A.bc_margin, d);
    }
    // 2D: margins from the x and the y faces that together hold every wall node
    // and every node with a program
    A.mx = A.px ? -1 : 0;
    A.my = A.py ? -1 : 0;
    for (uint32_t id = 0; lat == MPLB_D2Q9 && id < n; id++) {
        if (!map[id]) continue;
        const int x = (int)(id % (uint32_t)A.nx), y = (int)(id / (uint32_t)A.nx);
        const int dx = std::min(x, A.nx - 1 - x), dy = std::min(y, A.ny - 1 - y);
        if (dx <= A.mx || dy <= A.my) continue;
        if (dx < dy) A.mx = dx;
        else A.my = dy;
    }
    for (size_t q = 0; q < progs.size(); q++) A.prog[q] = progs[q];
    for (size_t p = 0; p < fp[1].size() && p < MPLB_MAX_PATCHES; p++) A.Twall[p] = fp[1][p].val[0];
    fc.has_bc = any;
    if (any) {
        if (cudaMalloc((void**)&fc.bcmap, n) != cudaSuccess) { fc.err = "cudaMalloc bcmap"; return MPLB_E_CUDA; }
        if (cudaMemcpyAsync(fc.bcmap, map.data(), n, cudaMemcpyHostToDevice, stream) != cudaSuccess) {
            fc.err = "copy bcmap";
            return MPLB_E_CUDA;
        }
        if (cudaStreamSynchronize(stream) != cudaSuccess) { fc.err = "copy bcmap"; return MPLB_E_CUDA; }
        *bytes += n;
    }
    A.bcmap = fc.bcmap;
    A.rho_a = A.gsum_a = nullptr;
    if (lat == MPLB_D2Q9 && model[1] == MPLB_MYMRT && P.g_update) {
        if (cudaMalloc((void**)&fc.my_scratch, 2 * (size_t)n * sizeof(double)) != cudaSuccess) {
            fc.err = "cudaMalloc myMRT scratch";
            return MPLB_E_CUDA;
        }
        *bytes += 2 * (size_t)n * sizeof(double);
        A.rho_a = fc.my_scratch;
        A.gsum_a = fc.my_scratch + n;
    }
    fc.lat = lat;
    fc.ncfg = lat == MPLB_D2Q9 ? N_CFG2 : N_CFG3;
    for (int c = 0; c < fc.ncfg; c++) {
        const TileCfg t = lat == MPLB_D2Q9 ? CFG2[c] : CFG3[c];
        if (t.tma) {
            fc.geom[c] = tma3_fits(A, any, t.tx, t.ty) ? resident_geometry(A, t.tx, t.ty, t.minb) : Geom{0, 0, 0, 0};
        } else if (t.table) {
            // two kernels that pull twice but have no ring, barrier or wrap arithmetic:
            // the better ones where boundary programs make a pull costly (us a step,
            // walls 97 x 61 x 83: 69 against 88 of the best tile; periodic 101 x 75 x
            // 90: 94 against 86; B200)
            fc.tab.nb = nb;
            fc.tab.onb = onb;
            fc.tab.bcmap = fc.bcmap;
            for (int q = 0; q < FUSED_MAX_PROGS; q++) fc.tab.prog[q] = A.prog[q];
            fc.geom[c] = Geom{1, 1, 1, (int)((n + 127) / 128)};
        } else if (t.march) {
            // (no march with a surface-tension term)
            const bool my = P.g_update && model[1] == MPLB_MYMRT && !P.st_on;
            fc.geom[c] = my ? march_geometry(A, mplb_march_resident(P.f_update != 0, any)) : Geom{0, 0, 0, 0};
        } else {
            fc.geom[c] = fused_geometry(lat, A, t.tx, t.ty);
        }
    }
    if (cudaMalloc((void**)&fc.kerr, sizeof(int)) != cudaSuccess) { fc.err = "cudaMalloc kernel flag"; return MPLB_E_CUDA; }
    if (cudaMallocHost((void**)&fc.kerr_host, sizeof(int)) != cudaSuccess) { fc.err = "cudaMallocHost kernel flag"; return MPLB_E_CUDA; }
    *fc.kerr_host = 0;
    if (cudaMemsetAsync(fc.kerr, 0, sizeof(int), stream) != cudaSuccess) { fc.err = "clear kernel flag"; return MPLB_E_CUDA; }
    *bytes += sizeof(int);
    A.kerr = fc.kerr;
    fc.cfg = 0;
    apply_geom(A, fc.geom[0]);
    fc.nblocks = fc.geom[0].nblocks;
    if (lat == MPLB_D3Q15 && fused_attributes() != cudaSuccess) {
        fc.err = "cannot raise the dynamic shared memory limit";
        return MPLB_E_CUDA;
    }
    return 0;
}

// The kernel error flag (0, or MPLB_KERR_WAIT after a bounded wait ran
// out): queue its copy to the pinned host int and its reset on the stream;
// after the caller's next synchronisation fused_kerr_value() holds it.
inline bool fused_queue_kerr(FusedConfig& fc, cudaStream_t s) {
    if (!fc.kerr) return true;
    return cudaMemcpyAsync(fc.kerr_host, fc.kerr, sizeof(int), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
           cudaMemsetAsync(fc.kerr, 0, sizeof(int), s) == cudaSuccess;
}
inline int fused_kerr_value(const FusedConfig& fc) { return fc.kerr_host ? *fc.kerr_host : 0; }

inline void fused_free(FusedConfig& fc) {
    if (fc.kerr) cudaFree(fc.kerr);
    fc.kerr = nullptr;
    if (fc.kerr_host) cudaFreeHost(fc.kerr_host);
    fc.kerr_host = nullptr;
    if (fc.bcmap) cudaFree(fc.bcmap);
    fc.bcmap = nullptr;
    if (fc.my_scratch) cudaFree(fc.my_scratch);
    fc.my_scratch = nullptr;
    if (fc.tab.psi) cudaFree(fc.tab.psi);
    fc.tab.psi = nullptr;
}


}  // namespace mplb
