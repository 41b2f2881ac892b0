// slice_emu.cpp — TEST INFRASTRUCTURE ONLY.
//
// Walks a component's sliced stream (ksim_b200/csrc/slice.cpp) on the CPU,
// one parameter row at a time with the roles the kernel gives each group, so
// the tests can check the stream against the oracle without a GPU.
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "image.h"
#include "slice.h"

using namespace ksim;

namespace {
std::string g_err;

// The row parities of a group (n rows) of the chunk at `base`.
void group(const uint8_t *base, uint32_t entry, int n, const std::vector<uint8_t> &v, int *r)
{
    const uint8_t *p = base + 16 * (entry & 0xFFFFu);
    const int slots = (int)(entry >> 16 & 0xFFu);
    for (int i = 0; i < n; ++i) {
        r[i] = p[4 * i] & 1;
        for (int k = 0; k < slots; ++k) r[i] ^= v[p[4 * n + 4 * n * (k / 4) + 4 * i + (k & 3)]];
    }
}
}  // namespace

extern "C" {

const char *slice_emu_error(void) { return g_err.c_str(); }

// info: ok, rows, max planes, chunks, bytes, terms, wide terms, terms with a global table
int slice_emu_info(const ksim_graph_desc *g, int n, int F, int64_t *info)
{
    HostImage img;
    const int st = build_image(g, n, F, img, g_err);
    if (st) return st;
    SliceImage s;
    build_slices(g, img, s);
    const int64_t v[5] = {s.ok, s.rows, s.max_planes, (int64_t)s.chunks.size(), (int64_t)s.bytes.size()};
    std::memcpy(info, v, sizeof(v));
    info[5] = info[6] = info[7] = 0;
    if (!s.ok) return 0;
    for (const ChunkDir &c : s.chunks)
        for (int t = 0; t < c.n_terms; ++t) {
            SliceTerm d;
            std::memcpy(&d, &s.bytes[c.off + SLICE_HEAD + t * sizeof(SliceTerm)], sizeof(d));
            info[5] += 1;
            info[6] += (d.flags & ST_WIDE) ? 1 : 0;
            info[7] += (d.flags & ST_BIG) ? 1 : 0;
        }
    return 0;
}

// Size of the stream built under a bound, or 0 if it does not fit.
int64_t slice_emu_bytes(const ksim_graph_desc *g, int n, int F, int64_t max_bytes)
{
    HostImage img;
    if (build_image(g, n, F, img, g_err)) return -1;
    SliceImage s;
    build_slices(g, img, s, (size_t)max_bytes);
    return s.ok ? (int64_t)s.bytes.size() : 0;
}

// Complex amplitude of graph gi for B explicit parameter rows.
int slice_emu_eval(const ksim_graph_desc *g, int n, int F, int gi, const uint8_t *params, int64_t B, int64_t P,
                   double *out)
{
    HostImage img;
    const int st = build_image(g, n, F, img, g_err);
    if (st) return st;
    SliceImage s;
    build_slices(g, img, s);
    if (!s.ok) return -1;
    for (int64_t b = 0; b < B; ++b) {
        std::vector<uint8_t> v((size_t)s.rows + 1, 0);
        for (int64_t j = 0; j < P && j < s.rows; ++j) v[j] = params[b * P + j] & 1;
        double sre = 0, sim = 0;
        for (const ChunkDir &c : s.chunks) {
            if (c.graph != gi) continue;
            const uint8_t *base = s.bytes.data() + c.off;
            for (int t = 0; t < c.n_terms; ++t) {
                SliceTerm d;
                SliceValue w;
                std::memcpy(&d, base + SLICE_HEAD + t * sizeof(SliceTerm), sizeof(d));
                const uint8_t *tabs = base + c.bytes;
                std::memcpy(&w, tabs + t * sizeof(SliceValue), sizeof(w));
                const uint8_t *list = base + 16 * d.list_off16;
                int r[8], kill = 0, K = 0, y = 0, z = 0, X = 0, S = 0;
                for (int q = 0; q < d.n_k + d.n_x1 + d.n_x0 + d.n_xp; ++q) {
                        uint32_t entry;
                        std::memcpy(&entry, list + 4 * q, 4);
                        const int m = SLICE_GROUP, role = (int)(entry >> 24 & 15u);
                        group(base, entry, m, v, r);
                        int sum = 0, prod = 0;
                        for (int i = 0; i < m; ++i) sum += r[i];
                        for (int i = 0; i < m; i += 2) prod += r[i] * r[i + 1];
                        switch (role) {
                        case SQ_KILL: kill |= sum; break;
                        case SQ_W1: K += sum; break;
                        case SQ_W2: K += 2 * sum; break;
                        case SQ_W4: K += 4 * sum; break;
                        case SQ_PPK: K += 4 * prod; break;
                        case SQ_PPX: S ^= prod & 1; break;
                        case SQ_N9:
                            for (int i = 0; i < m; i += 2) y += !r[i] && !r[i + 1];
                            z += prod;
                            break;
                        case SQ_X1: S ^= sum & 1; X += sum; break;
                        default: X += sum; break;
                        }
                    }
                K = (K + 4 * S) & 7;
                const int e = y + z;
                const int cls = (d.flags & ST_WIDE) ? tabs[16 * w.lut_off16 + (y | z << 4)] : e * (e + 1) / 2 + z;
                const int col = (d.flags & ST_EVEN) ? cls : 2 * cls + (K & 1);
                const size_t at = (size_t)(kill ? 0 : X + 1) * w.xs + (size_t)col * 16;
                const uint8_t *tab = (d.flags & ST_BIG) ? s.bytes.data() + 16 * (size_t)w.tab : tabs + w.tab;
                double re, im;
                std::memcpy(&re, tab + at, 8);
                std::memcpy(&im, tab + at + 8, 8);
                if (K & 2) { const double x = re; re = -im; im = x; }
                if (K & 4) { re = -re; im = -im; }
                sre += re;
                sim += im;
            }
        }
        out[2 * b] = sre;
        out[2 * b + 1] = sim;
    }
    return 0;
}

}  // extern "C"
