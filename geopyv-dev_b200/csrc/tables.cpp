// tables.cpp -- the per-radius template tables that the solve kernels read.
//
// Tables grow with the largest radius asked for.  Grown tables are built and
// filled in memory of their own and then take the old ones' place: a failure leaves
// the context with the tables that its radius says it has, and launches
// still in flight read the old ones until those are freed (which waits for them).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <string>
#include <vector>

#include "internal.h"
#include "run_window.h"

namespace gpv {
namespace {

// Device memory filled from a vector, released unless it replaces a buffer.
struct FreshBuf {
    DevBuf b;
    template <class T>
    int fill(const std::vector<T> &v) {
        if (int rc = b.ensure(v.size() * sizeof(T))) return rc;
        GPV_CUDA_TRY(cudaMemcpy(b.ptr, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
        GPV_CUDA_TRY(cudaStreamSynchronize(nullptr));  // solve streams do not wait for the copy's own
        return GPV_SUCCESS;
    }
    void replace(DevBuf &old) {
        std::swap(b, old);
        b.release();
    }
    ~FreshBuf() { b.release(); }
};

}  // namespace

struct short2_h {
    int16_t x, y;
};
constexpr int16_t kSlotEmpty = -32768;  // padding slot of a template row (see icgn_tile.cu)

// Circular local masks for radii 1..max_radius in the scan order of
// LocalMask::circle (src/masks.rs:69-109): rows y = -r..r, columns x = -r..r,
// kept when sqrt(x^2 + y^2) <= r (i.e. x^2 + y^2 <= r^2 for integers).
int ensure_tables(gpv_context *ctx, int max_radius) try {
    if (max_radius <= ctx->table_radius) return GPV_SUCCESS;
    if (max_radius > 4000) {
        set_error("radius above 4000 is not supported");
        return GPV_ERR_INVALID;
    }
    const int R1 = max_radius + 1;
    std::vector<short2_h> offs, slots;
    std::vector<int32_t> toff(R1, 0), tn(R1, 0), soff(R1, 0), sn(R1, 0), qoff(R1, 0), qn(R1, 0), nmax(R1, 0);
    for (int r = 1; r <= max_radius; r++) {
        toff[r] = (int32_t)offs.size();
        soff[r] = (int32_t)slots.size();
        for (int y = -r; y <= r; y++) {
            int row = 0;
            for (int x = -r; x <= r; x++)
                if (x * x + y * y <= r * r) {
                    offs.push_back({(int16_t)x, (int16_t)y});
                    slots.push_back({(int16_t)x, (int16_t)y});
                    row++;
                }
            // pad the template row to whole warps: a warp never straddles two rows
            while (row % 32) {
                slots.push_back({kSlotEmpty, (int16_t)y});
                row++;
            }
        }
        tn[r] = (int32_t)offs.size() - toff[r];
        sn[r] = (int32_t)slots.size() - soff[r];
    }
    // tiles: the disk covered by 8-wide x 4-high tiles, one per warp, slots in
    // tile order (4 rows of 8); with a window pitch of 8 mod 32 the 32 lanes
    // of a tile read 32 different shared-memory banks
    for (int r = 1; r <= max_radius; r++) {
        qoff[r] = (int32_t)slots.size();
        for (int y0 = -r; y0 <= r; y0 += 4) {
            int xmin = r + 1, xmax = -r - 1;
            for (int y = y0; y < y0 + 4 && y <= r; y++)
                for (int x = -r; x <= r; x++)
                    if (x * x + y * y <= r * r) { xmin = std::min(xmin, x); xmax = std::max(xmax, x); }
            for (int x0 = xmin; x0 <= xmax; x0 += 8)
                for (int ty = 0; ty < 4; ty++)
                    for (int tx = 0; tx < 8; tx++) {
                        const int x = x0 + tx, y = y0 + ty;
                        const bool in = y <= r && x * x + y * y <= r * r;
                        slots.push_back({in ? (int16_t)x : kSlotEmpty, (int16_t)y});
                    }
        }
        qn[r] = (int32_t)slots.size() - qoff[r];
        nmax[r] = std::max(std::max(tn[r], sn[r]), qn[r]);
    }
    // tab_off / tab_n: compact template tables, padded-row slot tables, tile slot tables
    std::vector<int32_t> to2(toff), tn2(tn);
    to2.insert(to2.end(), soff.begin(), soff.end());
    tn2.insert(tn2.end(), sn.begin(), sn.end());
    to2.insert(to2.end(), qoff.begin(), qoff.end());
    tn2.insert(tn2.end(), qn.begin(), qn.end());
    FreshBuf o, s, t, n;
    if (int rc = o.fill(offs)) return rc;
    if (int rc = s.fill(slots)) return rc;
    if (int rc = t.fill(to2)) return rc;
    if (int rc = n.fill(tn2)) return rc;
    o.replace(ctx->offs);
    s.replace(ctx->slots);
    t.replace(ctx->tab_off);
    n.replace(ctx->tab_n);
    ctx->h_tab_off.swap(toff);
    ctx->h_tab_n.swap(tn);
    ctx->h_slot_n.swap(nmax);  // the most slots any layout uses (per-block scratch)
    ctx->table_radius = max_radius;
    return GPV_SUCCESS;
} catch (const std::bad_alloc &) {
    set_error("no memory for the template tables");
    return GPV_ERR_NOMEM;
}

// Run tables for radii 1..max_radius: per run {dx (low 16 bits) | dy0 (high
// 16 bits), circle bits}, bands of kRunK rows from dy = -r, the last band
// moved up to end at dy = r (its rows already in the band above masked off);
// columns [-w, w] with w the widest circle row of the band.
int ensure_run_tables(gpv_context *ctx, int max_radius) try {
    if (max_radius <= ctx->run_table_radius) return GPV_SUCCESS;
    const int R1 = max_radius + 1;
    std::vector<int32_t> tab;  // pairs
    std::vector<int32_t> off(R1, 0), cnt(R1, 0);
    for (int r = 1; r <= max_radius; r++) {
        off[r] = (int32_t)(tab.size() / 2);
        int n = 0;
        for (int b0 = -r; b0 <= r; b0 += kRunK) {
            const int dy0 = (2 * r + 1 >= kRunK) ? std::min(b0, r - kRunK + 1) : -r;
            int w = -1;
            for (int j = 0; j < kRunK; j++) {
                const int y = dy0 + j;
                if (y < b0 || y > r) continue;
                // the row's exact integer half-width, then the band's widest
                int h = (int)std::floor(std::sqrt((double)(r * r - y * y)));
                while ((h + 1) * (h + 1) + y * y <= r * r) h++;
                while (h > 0 && h * h + y * y > r * r) h--;
                w = std::max(w, h);
            }
            for (int dx = -w; dx <= w; dx++) {
                uint32_t bits = 0;
                for (int j = 0; j < kRunK; j++) {
                    const int y = dy0 + j;
                    if (y >= b0 && y <= r && dx * dx + y * y <= r * r) bits |= 1u << j;
                }
                tab.push_back((int32_t)((uint32_t)(dx & 0xffff) | ((uint32_t)dy0 << 16)));
                tab.push_back((int32_t)bits);
                n++;
            }
        }
        cnt[r] = n;
    }
    // one buffer, one copy: run offsets, run counts, runs (8-byte aligned)
    std::vector<int32_t> all(off);
    all.insert(all.end(), cnt.begin(), cnt.end());
    all.insert(all.end(), tab.begin(), tab.end());
    FreshBuf b;
    if (int rc = b.fill(all)) return rc;
    b.replace(ctx->run_tab);
    ctx->h_run_n.swap(cnt);
    ctx->run_table_radius = max_radius;
    return GPV_SUCCESS;
} catch (const std::bad_alloc &) {
    set_error("no memory for the run tables");
    return GPV_ERR_NOMEM;
}

}  // namespace gpv
