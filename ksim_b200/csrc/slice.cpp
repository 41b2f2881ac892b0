// slice.cpp — builds the sliced term stream (slice.h) of a component.
#include "slice.h"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <iterator>

namespace ksim {
namespace {

typedef __int128 i128;

// Ring element times 2^e, basis (1, w, i, conj w).
struct El {
    i128 c[4];
    int e = 0;
};

El el(int64_t a, int64_t b, int64_t c, int64_t d) { return {{a, b, c, d}, 0}; }

El mul(const El &x, const El &y)
{
    El r;
    r.c[0] = x.c[0] * y.c[0] + x.c[1] * y.c[3] - x.c[2] * y.c[2] + x.c[3] * y.c[1];
    r.c[1] = x.c[0] * y.c[1] + x.c[1] * y.c[0] + x.c[2] * y.c[3] + x.c[3] * y.c[2];
    r.c[2] = x.c[0] * y.c[2] + x.c[1] * y.c[1] + x.c[2] * y.c[0] - x.c[3] * y.c[3];
    r.c[3] = x.c[0] * y.c[3] - x.c[1] * y.c[2] - x.c[2] * y.c[1] + x.c[3] * y.c[0];
    r.e = x.e + y.e;
    return r;
}

El rot1(const El &x)  // times w
{
    El r = x;
    r.c[0] = x.c[3]; r.c[1] = x.c[0]; r.c[2] = x.c[1]; r.c[3] = -x.c[2];
    return r;
}

El rot(El x, int k)
{
    for (k &= 7; k > 0; --k) x = rot1(x);
    return x;
}

// Take the common powers of two out of the coefficients.  False if one is
// beyond the range a product with a small factor keeps in 128 bits.
bool reduce(El &x)
{
    const i128 lim = (i128)1 << 90;
    i128 any = x.c[0] | x.c[1] | x.c[2] | x.c[3];
    if (any == 0) return true;
    while ((any & 1) == 0) {
        any = 0;
        for (i128 &v : x.c) {
            v >>= 1;
            any |= v;
        }
        ++x.e;
    }
    for (i128 v : x.c)
        if (v > lim || v < -lim) return false;
    return true;
}

// x lambda w^6 = x (w^5 + w^6 + w^7)  (lambda = 1 + w + conj w).
El step_lambda(const El &x)
{
    const i128 a = x.c[0], b = x.c[1], c = x.c[2], d = x.c[3];
    El r;
    r.c[0] = b + c - d;
    r.c[1] = c - a - d;
    r.c[2] = -(a + b + d);
    r.c[3] = a + b + c;
    r.e = x.e;
    return r;
}

bool same(const El &x, const El &y) { return x.e == y.e && std::equal(x.c, x.c + 4, y.c); }

// Complex value of x 2^(x.e + p2) as the reference casts it (zx_eval.hpp:
// 166-176); the scaling is exact or rounds once, as the reference's product.
void cast(const El &x, int64_t p2, double &re, double &im)
{
    const double SQh = 0.70710678118654752440;
    const double A = (double)(int64_t)x.c[0], B = (double)(int64_t)x.c[1];
    const double C = (double)(int64_t)x.c[2], D = (double)(int64_t)x.c[3];
    const double s1 = B + D, s2 = B - D;
    const double t1 = s1 * SQh, t2 = s2 * SQh;
    const int n = (int)std::max<int64_t>(-4000, std::min<int64_t>(4000, p2 + x.e));
    if (n >= -1022 && n <= 1023) {  // one product with the power of two, as the reference's
        const uint64_t bits = (uint64_t)(n + 1023) << 52;
        double scale;
        std::memcpy(&scale, &bits, 8);
        re = (A + t1) * scale;
        im = (C + t2) * scale;
    } else {
        re = std::ldexp(A + t1, n);
        im = std::ldexp(C + t2, n);
    }
}

// A parity row: its parameters (one bit each, so that nothing is allocated a
// row) and whether its parity is complemented.
struct Row {
    uint64_t bits[4] = {0, 0, 0, 0};
    uint32_t inv = 0;
    bool empty() const { return (bits[0] | bits[1] | bits[2] | bits[3]) == 0; }
    int weight() const
    {
        return __builtin_popcountll(bits[0]) + __builtin_popcountll(bits[1]) + __builtin_popcountll(bits[2]) +
               __builtin_popcountll(bits[3]);
    }
};
static_assert(SLICE_MAX_ROWS <= 256, "Row");

Row make_row(const uint8_t *m, int P, uint32_t inv)
{
    Row r;
    r.inv = inv & 1u;
    int j = 0;
    for (; j + 8 <= P; j += 8) {  // eight mask bytes (0 or 1) to eight bits
        uint64_t x;
        std::memcpy(&x, m + j, 8);
        r.bits[j >> 6] |= (x * 0x0102040810204080ull >> 56) << (j & 63);
    }
    for (; j < P; ++j) r.bits[j >> 6] |= (uint64_t)(m[j] & 1u) << (j & 63);
    return r;
}

Row flip(Row r)
{
    r.inv ^= 1u;
    return r;
}

Row xor_rows(const Row &a, const Row &b)
{
    Row r;
    r.inv = a.inv ^ b.inv;
    for (int i = 0; i < 4; ++i) r.bits[i] = a.bits[i] ^ b.bits[i];
    return r;
}

// A row's parameters, in order; returns how many.
int row_indices(const Row &r, uint8_t *out)
{
    int n = 0;
    for (int i = 0; i < 4; ++i)
        for (uint64_t x = r.bits[i]; x; x &= x - 1) out[n++] = (uint8_t)(64 * i + __builtin_ctzll(x));
    return n;
}

// A PhasePairs factor as one of the kinds of slice.h times w^k.
enum Kind { K_ZERO, K_TWO, K_22, K_P, K_Q, K_B, K_L0, K_L1 };
const El kTwo = el(2, 0, 0, 0), k22 = el(2, 0, 2, 0), kP = el(1, 2, -1, 0), kQ = el(1, -2, -1, 0),
         kB = el(1, 0, 1, 0), kKappa = el(1, -1, 1, -1), kLam = el(1, 1, 0, 1), kLamInv = el(-1, 1, 0, 1);

bool find_kind(int a, int b, Kind &kind, int &k)
{
    const El one = el(1, 0, 0, 0);
    const El u = rot(one, a), v = rot(one, b), x = rot(one, a + b);
    El f;
    for (int i = 0; i < 4; ++i) f.c[i] = one.c[i] + u.c[i] + v.c[i] - x.c[i];
    if ((f.c[0] | f.c[1] | f.c[2] | f.c[3]) == 0) {
        kind = K_ZERO;
        k = 0;
        return true;
    }
    const struct { Kind kind; El el; } cand[] = {{K_TWO, kTwo}, {K_22, k22}, {K_P, kP}, {K_Q, kQ}, {K_B, kB},
                                                 {K_L0, kKappa}, {K_L1, mul(kKappa, kLam)}};
    for (const auto &c : cand)
        for (k = 0; k < 8; ++k)
            if (same(f, rot(c.el, k))) {
                kind = c.kind;
                return true;
            }
    return false;
}

// The kinds of all 64 (alpha, beta) pairs.
struct KindTable {
    Kind kind[8][8];
    int k[8][8];
    bool ok[8][8];
    KindTable()
    {
        for (int a = 0; a < 8; ++a)
            for (int b = 0; b < 8; ++b) ok[a][b] = find_kind(a, b, kind[a][b], k[a][b]);
    }
};

bool classify(int a, int b, Kind &kind, int &k)
{
    static const KindTable t;
    kind = t.kind[a][b];
    k = t.k[a][b];
    return t.ok[a][b];
}

// A term's rows by role.
struct TermRows {
    std::vector<Row> kill, w1, w2, x1, x0;
    std::vector<Row> pp, n9;  // pairs
    Row w4;
    int k0 = 0;          // constant part of K
    int n_two = 0, n_22 = 0, n_8 = 0;

    void weight(const Row &r, int w)
    {
        switch (w & 7) {
        case 1: w1.push_back(r); break;
        case 2: w2.push_back(r); break;
        case 3: weight(r, 7); weight(r, 4); break;
        case 4:
            w4 = xor_rows(w4, r);
            break;
        case 5: weight(r, 1); weight(r, 4); break;
        case 6: w2.push_back(flip(r)); k0 += 6; break;
        case 7: w1.push_back(flip(r)); k0 += 7; break;
        default: break;
        }
    }
};

// A group of SLICE_GROUP rows of one role: 4 bytes a row of complement masks,
// then index units: four slots of each row (a byte is a parameter row; the rows
// with fewer name the zero row).
struct Group {
    std::vector<uint8_t> bytes;
    uint32_t slots = 0;  // index slots a row
    uint32_t role = 0;
    double cost() const { return 3.0 * slots + 8.0; }
};

Group make_group(const Row *const *rows, int n, int zero_row)
{
    Group g;
    uint8_t idx[SLICE_GROUP][256];
    int len[SLICE_GROUP], slots = 1;
    for (int r = 0; r < n; ++r) {
        len[r] = row_indices(*rows[r], idx[r]);
        slots = std::max(slots, len[r]);
    }
    g.slots = (uint32_t)slots;
    g.bytes.assign((size_t)n * (4 + (size_t)(slots + 3) / 4 * 4), (uint8_t)zero_row);
    for (int r = 0; r < n; ++r) std::memset(&g.bytes[4 * (size_t)r], rows[r]->inv ? 0xFF : 0, 4);
    for (int r = 0; r < n; ++r)
        for (int k = 0; k < len[r]; ++k) g.bytes[(size_t)(4 * n + 4 * n * (k / 4) + 4 * r + (k & 3))] = idx[r][k];
    return g;
}

// Rows of one role, heaviest first (a group runs as many index slots as its
// longest row), `step` rows kept together, padded with pad0 / zero rows.
std::vector<Group> make_groups(const std::vector<Row> &rows, int step, const Row &pad0, int zero_row)
{
    const Row zero;
    std::vector<size_t> order;
    for (size_t i = 0; i < rows.size(); i += (size_t)step) order.push_back(i);
    std::vector<int> weight(rows.size());
    for (size_t i = 0; i < rows.size(); ++i) weight[i] = rows[i].weight();
    if (step == 2)
        for (size_t i = 0; i < rows.size(); i += 2) weight[i] = std::max(weight[i], weight[i + 1]);
    if (order.size() > 1)
        std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) { return weight[x] > weight[y]; });
    std::vector<const Row *> seq;
    seq.reserve(rows.size() + 3);
    for (size_t i : order)
        for (int k = 0; k < step; ++k) seq.push_back(&rows[i + (size_t)k]);
    while (seq.size() % SLICE_GROUP) seq.push_back(step == 1 || (seq.size() & 1u) ? &zero : &pad0);
    std::vector<Group> out;
    for (size_t i = 0; i < seq.size();) {
        out.push_back(make_group(&seq[i], SLICE_GROUP, zero_row));
        i += SLICE_GROUP;
    }
    return out;
}

struct TermOutBytes {
    SliceTerm d;
    SliceValue v;
    std::vector<Group> groups;  // role by role
    size_t rows_bytes() const
    {
        size_t n = (4 * groups.size() + 15) / 16 * 16;
        for (const Group &x : groups) n += x.bytes.size();
        return n;
    }
    std::vector<uint8_t> lut, tab;
    int planes = 2;
};

// Rows and table of one term; false if it does not qualify.
bool build_term(const ksim_graph_desc &g, int t, int zero_row, TermOutBytes &o)
{
    const int P = g.P;
    TermRows R;
    El base = el(1, 0, 0, 0);
    int n1 = 0, n3 = 0;
    const int cnp = std::max(0, g.np_counts[t]), cph = std::max(0, g.ph_counts[t]);
    for (int c = 0; c < cnp; ++c) {
        const size_t ci = (size_t)t * g.Tnp + c;
        const uint32_t ph = g.np_phases[ci] & 7u;
        const Row r = make_row(g.np_params + ci * P, P, ph >> 2);
        switch (ph & 3u) {
        case 0:
            R.kill.push_back(r);
            base.e += 1;  // the factor of a live shot: 2
            break;
        case 1:
            R.x1.push_back(flip(r));
            base = mul(base, el(1, 1, 0, 0));
            ++n1;
            break;
        case 2:
            R.weight(r, 6);
            base = mul(base, el(1, 0, 1, 0));
            break;
        default:
            R.x0.push_back(r);
            base = mul(base, el(1, 0, 0, -1));
            ++n3;
            break;
        }
        if (!reduce(base)) return false;
    }
    // 6 (m1 + m3) = 6 (X - n1) + 4 m1, and the parity of the complemented
    // class-1 rows is m1 + n1
    R.k0 += -6 * n1 + 4 * n1;
    for (int c = 0; c < g.Thp; ++c) {
        const size_t ci = (size_t)t * g.Thp + c;
        R.weight(make_row(g.hp_params + ci * P, P, 0), g.hp_coeffs[ci] & 7);
    }
    for (int c = 0; c < g.Tpp; ++c) {
        const size_t ci = (size_t)t * g.Tpp + c;
        const Row psi = make_row(g.pp_psi_p + ci * P, P, g.pp_psi_c[ci]);
        const Row phi = make_row(g.pp_phi_p + ci * P, P, g.pp_phi_c[ci]);
        if ((psi.empty() && !psi.inv) || (phi.empty() && !phi.inv)) continue;
        R.pp.push_back(psi);
        R.pp.push_back(phi);
    }
    for (int c = 0; c < cph; ++c) {
        const size_t ci = (size_t)t * g.Tph + c;
        const uint32_t a = g.ph_alpha[ci] & 7u, b = g.ph_beta[ci] & 7u;
        Row sa = make_row(g.ph_alpha_p + ci * P, P, a >> 2), sb = make_row(g.ph_beta_p + ci * P, P, b >> 2);
        Kind kind[4];
        int k[4];
        for (int s = 0; s < 4; ++s) {
            if (!classify((int)(a & 3u) + 4 * (s & 1), (int)(b & 3u) + 4 * (s >> 1), kind[s], k[s])) return false;
            if (kind[s] == K_L1) k[s] += 2;  // w^(6X) is in the tables: lambda^1 carries w^6 there
        }
        if (kind[1] == K_ZERO && kind[2] == K_ZERO) {  // signs differ: zero
            R.kill.push_back(xor_rows(sa, sb));
            R.weight(sa, k[3] - k[0] + 8);
            R.k0 += k[0];
            R.n_22 += 1;
            continue;
        }
        const int wa = (k[1] - k[0] + 8) & 7, wb = (k[2] - k[0] + 8) & 7, wab = (k[3] - k[1] - k[2] + k[0] + 16) & 7;
        if (wab != 0 && wab != 4) return false;
        if (wab) {
            R.pp.push_back(sa);
            R.pp.push_back(sb);
        }
        R.k0 += k[0];
        R.weight(sa, wa);
        R.weight(sb, wb);
        if (kind[0] == K_TWO && kind[1] == K_TWO && kind[2] == K_TWO && kind[3] == K_TWO) {
            R.n_two += 1;
        } else if (kind[0] == K_L1 && kind[3] == K_L1 && kind[1] == K_L0 && kind[2] == K_L0) {
            R.x0.push_back(flip(xor_rows(sa, sb)));
            R.n_8 += 1;
        } else if (kind[1] == K_B && kind[2] == K_B &&
                   ((kind[0] == K_P && kind[3] == K_Q) || (kind[0] == K_Q && kind[3] == K_P))) {
            // rows such that both clear is p and both set is q
            R.n9.push_back(kind[0] == K_P ? sa : flip(sa));
            R.n9.push_back(kind[0] == K_P ? sb : flip(sb));
        } else {
            return false;
        }
    }
    R.k0 += (R.w4.inv ? 4 : 0) + (int)(g.pf_phase_idx[t] & 7u);
    const int n9 = (int)R.n9.size() / 2, nx = n1 + n3 + R.n_8;
    if (nx > 126 || n9 > 15) return false;
    const bool wide = n9 > 4, even = R.w1.empty();

    SliceTerm &d = o.d;
    std::memset(&d, 0, sizeof(d));
    std::memset(&o.v, 0, sizeof(o.v));
    d.flags = (uint16_t)((wide ? ST_WIDE : 0u) | (even ? ST_EVEN : 0u));
    o.planes = wide ? 3 : 2;
    std::vector<Group> role[SQ_ROLES];
    role[SQ_KILL] = make_groups(R.kill, 1, Row(), zero_row);
    role[SQ_W1] = make_groups(R.w1, 1, Row(), zero_row);
    role[SQ_W2] = make_groups(R.w2, 1, Row(), zero_row);
    // the weight-4 row's parameters, spread over the rows of one group
    std::vector<Row> w4(R.w4.empty() ? 0 : SLICE_GROUP);
    uint8_t idx4[256];
    const int n4 = row_indices(R.w4, idx4);
    for (int i = 0; i < n4; ++i) w4[(size_t)i % SLICE_GROUP].bits[idx4[i] >> 6] |= 1ull << (idx4[i] & 63);
    role[SQ_W4] = make_groups(w4, 1, Row(), zero_row);
    Row ones;  // pads the p / q pairs: one row set, one clear
    ones.inv = 1;
    role[SQ_N9] = make_groups(R.n9, 2, ones, zero_row);
    role[SQ_X1] = make_groups(R.x1, 1, Row(), zero_row);
    role[SQ_X0] = make_groups(R.x0, 1, Row(), zero_row);
    // the pair products enter K's bit 2 or its other half S: they go to
    // whichever half of the term has less to do
    double cost_k = 0, cost_x = 0;
    for (int i : {SQ_W1, SQ_W2, SQ_W4, SQ_N9})
        for (const Group &x : role[i]) cost_k += x.cost();
    for (int i : {SQ_X1, SQ_X0, SQ_KILL})
        for (const Group &x : role[i]) cost_x += x.cost();
    for (Group &x : make_groups(R.pp, 2, Row(), zero_row)) {
        double &c = cost_k <= cost_x ? cost_k : cost_x;
        c += x.cost();
        role[&c == &cost_k ? SQ_PPK : SQ_PPX].push_back(std::move(x));
    }
    for (uint32_t i = 0; i < SQ_ROLES; ++i)
        for (Group &x : role[i]) {
            x.role = i;
            if (x.slots > 255u) return false;
            (i < SQ_X1 ? d.n_k : i == SQ_X1 ? d.n_x1 : i == SQ_X0 ? d.n_x0 : d.n_xp) += 1;
            o.groups.push_back(std::move(x));
        }

    // classes (y, z) in the order of y + z, then z: class e (e + 1) / 2 + z
    std::vector<std::pair<int, int>> cls;
    for (int e = 0; e <= n9; ++e)
        for (int z = 0; z <= e; ++z) cls.push_back({e - z, z});
    if (wide) {
        o.lut.assign(256, 0);
        for (size_t c = 0; c < cls.size(); ++c) o.lut[(size_t)(cls[c].first | cls[c].second << 4)] = (uint8_t)c;
    }
    const int n_par = even ? 1 : 2;
    const size_t xs = cls.size() * (size_t)n_par * 16;
    o.v.xs = (uint16_t)xs;
    o.tab.assign(xs * (size_t)(nx + 2), 0);

    base.e += R.n_two;
    for (int i = 0; i < R.n_22; ++i) {
        base = mul(base, k22);
        if (!reduce(base)) return false;
    }
    for (int i = 0; i < R.n_8; ++i) {
        base = mul(base, kKappa);
        if (!reduce(base)) return false;
    }
    for (int i = 0; i < n1; ++i) {  // X = 0: lambda^-n1
        base = mul(base, kLamInv);
        if (!reduce(base)) return false;
    }
    const int32_t *ff = g.pf_floatfactor + 4 * (size_t)t;
    base = mul(rot(base, ((R.k0 % 8) + 8) & 7), el(ff[0], ff[1], ff[2], ff[3]));
    if (!reduce(base)) return false;
    const int64_t p2 = g.pf_power2[t];
    double ar = 1, ai = 0;
    if (g.pf_has_approx) {
        ar = g.pf_approx_f32[2 * (size_t)t];
        ai = g.pf_approx_f32[2 * (size_t)t + 1];
        // a dead term's 0 times an infinity or NaN is NaN, but its table row is zero
        if (!std::isfinite(ar) || !std::isfinite(ai)) return false;
    }
    for (size_t ci = 0; ci < cls.size(); ++ci) {
        const int y = cls[ci].first, z = cls[ci].second;
        El v = base;
        for (int i = 0; i < n9; ++i) {
            v = mul(v, i < y ? kP : i < y + z ? kQ : kB);
            if (!reduce(v)) return false;
        }
        for (int X = 0; X <= nx; ++X) {
            if (X) {
                v = step_lambda(v);
                if (!reduce(v)) return false;
            }
            for (i128 c : v.c)
                if (c > ((i128)1 << 62) || c < -((i128)1 << 62)) return false;
            El w = v;
            for (int r = 0; r < n_par; ++r) {
                double re, im;
                cast(w, p2, re, im);
                if (g.pf_has_approx) {
                    const double a = re * ar, b = im * ai, c = re * ai, e = im * ar;
                    re = a - b;
                    im = c + e;
                }
                const size_t at = (size_t)(X + 1) * xs + (ci * (size_t)n_par + (size_t)r) * 16;
                std::memcpy(&o.tab[at], &re, 8);
                std::memcpy(&o.tab[at + 8], &im, 8);
                w = rot1(w);
            }
        }
    }
    return true;
}

}  // namespace

void build_slices(const ksim_graph_desc *gs, const HostImage &img, SliceImage &out, size_t max_bytes)
{
    out = SliceImage();
    int rows = img.F + img.n_out;
    for (int k = 0; k < img.n_graphs; ++k) {
        rows = std::max(rows, gs[k].P);
        for (uint8_t f : img.term_proof[k])
            if (f != TP_ALL) return;
    }
    if (rows > SLICE_MAX_ROWS) return;
    out.rows = rows;
    std::vector<uint8_t> big;  // tables kept in global memory, behind the chunks
    struct BigRef { size_t desc; size_t off; };
    std::vector<BigRef> refs;
    auto pad = [](std::vector<uint8_t> &b, size_t to) { while (b.size() % to) b.push_back(0); };
    for (int k = 0; k < img.n_graphs; ++k) {
        const ksim_graph_desc &g = gs[k];
        int t = 0;
        TermOutBytes o;  // term t, once built
        bool built = false;
        do {
            // the terms of this chunk: as many as fit the slots and the planes
            std::vector<TermOutBytes> terms;
            size_t rows_bytes = SLICE_HEAD, tab_bytes = 0;
            int planes = 0;
            for (; t < g.G; ++t) {
                if (!built) {
                    o = TermOutBytes();
                    if (!build_term(g, t, rows, o)) return;
                    built = true;
                }
                const bool is_big = o.tab.size() > (size_t)SLICE_BIG_TABLE;
                if (is_big) o.d.flags |= ST_BIG;
                const size_t need_r = sizeof(SliceTerm) + o.rows_bytes();
                const size_t need_t = sizeof(SliceValue) + o.lut.size() + (is_big ? 0 : o.tab.size());
                if (SLICE_HEAD + need_r > (size_t)SLICE_SLOT) return;
                if (rows_bytes + need_r > (size_t)SLICE_SLOT || tab_bytes + need_t > (size_t)SLICE_TABLES ||
                    planes + o.planes > SLICE_MAX_PLANES || terms.size() == (size_t)SLICE_MAX_TERMS)
                    break;
                o.d.plane = o.v.plane = (uint16_t)planes;
                o.v.flags = o.d.flags;
                rows_bytes += need_r;
                tab_bytes += need_t;
                planes += o.planes;
                terms.push_back(std::move(o));
                built = false;
            }
            ChunkDir c = {};
            c.off = (int64_t)out.bytes.size();
            c.graph = k;
            c.n_terms = (int32_t)terms.size();
            c.end_of_graph = t >= g.G ? 1 : 0;
            std::vector<uint8_t> body(SLICE_HEAD + sizeof(SliceTerm) * terms.size(), 0);
            for (size_t i = 0; i < terms.size(); ++i) {
                TermOutBytes &o = terms[i];
                o.d.list_off16 = (uint16_t)(body.size() / 16);
                size_t at = body.size() + (4 * o.groups.size() + 15) / 16 * 16;
                for (const Group &x : o.groups) {
                    const uint32_t e = (uint32_t)(at / 16) | x.slots << 16 | x.role << 24;
                    body.insert(body.end(), (const uint8_t *)&e, (const uint8_t *)&e + 4);
                    at += x.bytes.size();
                }
                pad(body, 16);
                for (const Group &x : o.groups) body.insert(body.end(), x.bytes.begin(), x.bytes.end());
                std::memcpy(&body[SLICE_HEAD + i * sizeof(SliceTerm)], &o.d, sizeof(SliceTerm));
            }
            c.bytes = (int32_t)body.size();
            // (never empty: a copy is at least 16 bytes)
            std::vector<uint8_t> tabs(sizeof(SliceValue) * std::max<size_t>(1, terms.size()), 0);
            for (size_t i = 0; i < terms.size(); ++i) {
                TermOutBytes &o = terms[i];
                o.v.lut_off16 = (uint16_t)(tabs.size() / 16);
                tabs.insert(tabs.end(), o.lut.begin(), o.lut.end());
                if (o.d.flags & ST_BIG) {
                    refs.push_back({(size_t)c.off + body.size() + i * sizeof(SliceValue), big.size()});
                    big.insert(big.end(), o.tab.begin(), o.tab.end());
                } else {
                    o.v.tab = (uint32_t)tabs.size();
                    tabs.insert(tabs.end(), o.tab.begin(), o.tab.end());
                }
                std::memcpy(&tabs[i * sizeof(SliceValue)], &o.v, sizeof(SliceValue));
            }
            c.pad0 = (int32_t)tabs.size();
            out.bytes.insert(out.bytes.end(), body.begin(), body.end());
            out.bytes.insert(out.bytes.end(), tabs.begin(), tabs.end());
            out.max_planes = std::max(out.max_planes, planes);
            out.chunks.push_back(c);
            if (out.bytes.size() + big.size() > max_bytes) return;
        } while (t < g.G);
    }
    for (size_t i = 0; i < out.chunks.size(); ++i) {
        const ChunkDir &c = out.chunks[i];
        SliceChunk h = {};
        h.n_terms = (uint16_t)c.n_terms;
        h.end_of_graph = (uint16_t)c.end_of_graph;
        h.graph = (uint32_t)c.graph;
        if (i + SLICE_AHEAD < out.chunks.size()) {
            const ChunkDir &a = out.chunks[i + SLICE_AHEAD];
            h.ahead_bytes = (uint32_t)a.bytes;
            h.ahead_off16 = (uint32_t)(a.off / 16);
        }
        if (i + 1 < out.chunks.size()) {
            const ChunkDir &a = out.chunks[i + 1];
            h.tab_bytes = (uint32_t)a.pad0;
            h.tab_off16 = (uint32_t)((a.off + a.bytes) / 16);
        }
        std::memcpy(&out.bytes[(size_t)c.off], &h, sizeof(h));
    }
    pad(out.bytes, 16);
    const size_t at = out.bytes.size();
    for (const BigRef &r : refs) {
        const uint32_t off = (uint32_t)((at + r.off) / 16);
        std::memcpy(&out.bytes[r.desc + offsetof(SliceValue, tab)], &off, 4);
    }
    out.bytes.insert(out.bytes.end(), big.begin(), big.end());
    if (out.bytes.empty()) out.bytes.resize(16, 0);
    if (out.bytes.size() / 16 > 0xFFFFFFFFull) return;
    out.ok = true;
}

}  // namespace ksim
