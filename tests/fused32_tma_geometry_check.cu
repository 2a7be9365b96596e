// Host-only check of the TMA-staged D3Q15 kernels' staging (no GPU needed), FP64
// and FP32: tensor-copy boxes aligned, shared memory, and the stage after the
// tensor copies (zeros outside the lattice) and the copies of the wrapped parts
// holds, for every slot and population, the node the pull reads; every node is
// collided by exactly one thread.  Prints "OK <cases>" or the first violation.
#include <cstdio>
#include <cstring>
#include <vector>
#include "../multiphaselb_b200/csrc/fused32_tma.cuh"
#include "../multiphaselb_b200/csrc/fused_tma.cuh"

using namespace mplb;

static int fails = 0;
#define REQUIRE(c, ...) do { if (!(c) && fails++ < 10) { printf("FAIL %s:%d ", __FILE__, __LINE__); printf(__VA_ARGS__); printf("\n"); } } while (0)

// V: element type of the populations; boxes reach HX columns (16 bytes) past the tile.
template <class V, int TX, int TY, int MINB>
void check(int nx, int ny, int nz) {
    using L = D3Q15T;
    constexpr int HX = 16 / sizeof(V), BX = TX + 2 * HX, TBX = TX + 4, BY = TY + 2, NT = TX * TY;
    FusedArgs A{};
    A.nx = nx; A.ny = ny; A.nz = nz; A.px = A.py = A.pz = 1;
    if (sizeof(V) == 8 ? !tma3_fits(A, false, TX, TY) : !tma3_fits32(nx, ny, nz, 1, 1, 1, false, TX, TY)) return;
    const Geom gm = resident_geometry(A, TX, TY, MINB);
    if constexpr (sizeof(V) == 8) {
        using G = TmaTile<TX, TY>;
        REQUIRE(G::BX == BX && G::BY == BY && (2 * G::NSTAGE + 1) * 8 + 4 <= G::HEAD && G::SMEM <= 227 * 1024, "layout");
    } else {
        using G = TmaTile32<TX, TY>;
        REQUIRE(G::BX == BX && G::TBX == TBX && G::BY == BY && (2 * G::NSTAGE + 1) * 8 + 4 <= G::HEAD, "layout");
        REQUIRE(G::BOX_PITCH % 128 == 0 && G::BOX_PITCH >= G::BOX_BYTES && G::T_PITCH % 128 == 0 && G::T_PITCH >= G::T_BYTES, "pitch");
        REQUIRE((size_t)G::HEAD + (size_t)G::NSTAGE * G::STAGE_BYTES + (size_t)G::NPSI * G::EY * G::EX * 8 + 127 <= G::SMEM, "smem");
        REQUIRE(G::SMEM <= 227 * 1024, "smem limit");
    }
    const int64_t n = (int64_t)nx * ny * nz;
    std::vector<V> f(15 * n);
    std::vector<double> T(n);
    for (int64_t i = 0; i < 15 * n; i++) f[i] = (V)(i + 1);
    for (int64_t i = 0; i < n; i++) T[i] = (double)(i + 1);
    std::vector<int> owned(n, 0);
    std::vector<V> box(15 * BX * BY);
    std::vector<double> tb(TBX * BY);
    auto put = [&](unsigned char* dst, const unsigned char* src, size_t bytes) {
        const size_t db = (size_t)(dst - (unsigned char*)box.data()), dt = (size_t)(dst - (unsigned char*)tb.data());
        const size_t sb = (size_t)(src - (unsigned char*)f.data()), st = (size_t)(src - (unsigned char*)T.data());
        const bool okb = db + bytes <= box.size() * sizeof(V) && sb + bytes <= f.size() * sizeof(V) && db % 16 == 0 && sb % 16 == 0;
        const bool okt = dt + bytes <= tb.size() * 8 && st + bytes <= T.size() * 8 && dt % 16 == 0 && st % 16 == 0;
        REQUIRE((okb || okt) && bytes % 16 == 0 && bytes > 0, "copy of %zu bytes out of place", bytes);
        if (okb || okt) std::memcpy(dst, src, bytes);
    };
    const int tiles = gm.tiles_x * gm.tiles_y;
    for (int b = 0; b < gm.nblocks; b++) {
        const int col = b % tiles, chunk = b / tiles;
        const int x0 = (col % gm.tiles_x) * TX, y0 = (col / gm.tiles_x) * TY;
        const int z0 = chunk * gm.zchunk, z1 = std::min(z0 + gm.zchunk, nz);
        REQUIRE(z0 < nz, "empty chunk");
        const bool face = x0 == 0 || x0 + TX == nx || y0 == 0 || y0 + TY == ny;
        REQUIRE((x0 - HX) * (int)sizeof(V) % 16 == 0 && (x0 - 2) * 8 % 16 == 0, "x of a tensor copy");
        for (int p = z0 - 1; p <= z1; p++) {
            if (p > z0 && p < z1 - 1) goto collided;  // first, last and halo planes stand for the rest
            for (int k = 0; k < 16; k++)
                for (int iy = 0; iy < BY; iy++)
                    for (int ix = 0; ix < (k < 15 ? BX : TBX); ix++) {
                        const int x = (k < 15 ? x0 - HX : x0 - 2) + ix, y = y0 - 1 - (k < 15 ? cyk<L>(k) : 0) + iy;
                        const int z = wrap_any(p - (k < 15 ? czk<L>(k) : 0), nz);
                        const bool in = x >= 0 && x < nx && y >= 0 && y < ny;
                        REQUIRE(z >= 0 && z < nz, "plane");
                        const int64_t at = (int64_t)x + (int64_t)nx * (y + (int64_t)ny * z);
                        if (k < 15) box[(k * BY + iy) * BX + ix] = in ? f[k * n + at] : (V)0;
                        else tb[iy * TBX + ix] = in ? T[at] : 0.0;
                    }
            if (face)
                for (int tid = 0; tid < NT; tid++)
                    patch_wrapped<TX, TY, 16>(tid, NT, x0, y0, nx, ny, [](int k) { return k < 15 ? cyk<L>(k) : 0; },
                        [&](int k, int iy, int y, unsigned char*& dst, const unsigned char*& src, int& es) {
                            REQUIRE(k < 16 && iy >= 0 && iy < BY && y >= 0 && y < ny, "row");
                            const int64_t row = (int64_t)nx * (y + (int64_t)ny * wrap_any(p - (k < 15 ? czk<L>(k) : 0), nz));
                            es = k < 15 ? (int)sizeof(V) : 8;
                            dst = k < 15 ? (unsigned char*)&box[(k * BY + iy) * BX] : (unsigned char*)&tb[iy * TBX];
                            src = k < 15 ? (const unsigned char*)&f[k * n + row] : (const unsigned char*)&T[row];
                        },
                        [&](unsigned char* dst, const unsigned char* src) { put(dst, src, 16); },
                        [&](unsigned char* dst, const unsigned char* src, int bytes) { put(dst, src, (size_t)bytes); });
            for (int ey = 0; ey < BY; ey++)
                for (int ex = 0; ex < TX + 2; ex++) {
                    const int sx = wrap_any(x0 - 1 + ex, nx), sy = wrap_any(y0 - 1 + ey, ny), sz = wrap_any(p, nz);
                    for (int k = 0; k < 15; k++) {
                        const int64_t src = pull_src(nx, ny, nz, 1, 1, 1, sx, sy, sz, cxk<L>(k), cyk<L>(k), czk<L>(k));
                        REQUIRE(box[(k * BY + ey) * BX + ex + HX - 1 - cxk<L>(k)] == f[k * n + src], "slot (%d,%d) k %d of tile (%d,%d)", ex, ey, k, x0, y0);
                    }
                    REQUIRE(tb[ey * TBX + ex + 1] == T[sx + (int64_t)nx * (sy + (int64_t)ny * sz)], "T of slot");
                }
        collided:
            if (p - 1 >= z0)
                for (int t = 0; t < NT; t++) owned[(size_t)(x0 + t % TX) + (size_t)nx * ((size_t)(y0 + t / TX) + (size_t)ny * (p - 1))]++;
        }
    }
    for (int64_t i = 0; i < n; i++) REQUIRE(owned[i] == 1, "node %lld collided %d times", (long long)i, owned[i]);
}

int main() {
    const int dims[][3] = {{32, 8, 2}, {32, 4, 5}, {64, 8, 3}, {64, 16, 9}, {96, 40, 3}, {128, 24, 7}, {192, 48, 2}, {32, 16, 17}, {160, 12, 11}};
    int cases = 0;
    for (auto& d : dims) {
        check<double, 64, 8, 1>(d[0], d[1], d[2]);
        check<double, 32, 8, 2>(d[0], d[1], d[2]);
        check<double, 32, 4, 3>(d[0], d[1], d[2]);
        check<double, 32, 16, 1>(d[0], d[1], d[2]);
        check<float, 64, 8, 1>(d[0], d[1], d[2]);
        check<float, 32, 8, 2>(d[0], d[1], d[2]);
        check<float, 32, 4, 5>(d[0], d[1], d[2]);
        check<float, 64, 4, 3>(d[0], d[1], d[2]);
        check<float, 32, 16, 1>(d[0], d[1], d[2]);
        cases++;
    }
    if (fails) { printf("FAILED %d checks\n", fails); return 1; }
    printf("OK %d\n", cases);
    return 0;
}
