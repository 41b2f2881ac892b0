// slice_tile.cuh — the per-CTA sampling loop over a sliced stream (slice.h).
//
// The parameter vector of a tile's shots lives bit-sliced in shared memory:
// one row of words per parameter, bit = shot.  Per chunk of terms the CTA
// runs two passes:
//   rows    a warp takes one half of a term (its K roles or its X roles): L
//           lanes cover the tile's shots, 64 each, and the 32 / L lane groups
//           share the groups of four rows of every role.  A lane forms parity
//           rows as XORs of a few parameter words and adds them into
//           bit-sliced counters (carry-save adders); the lane groups' counters
//           are added over shuffles, and the eight result planes become one
//           byte per shot by in-register 8 x 8 bit transposes;
//   values  a thread takes its S shots: two result bytes a term give the
//           table entry (a complex double) and its rotation by i^k; the
//           entries are added in term order.
// At a graph's end each thread makes its Bernoulli draws and the warp writes
// the sampled output's row with ballots (kokkos_sim.cpp:214-230).
//
// Chunks are staged by TMA bulk copies with bounded waits, the rows of a chunk
// in a ring of two slots, its tables in one slot: the tables' copy is issued
// when the chunk before is done and hides behind the rows pass, which needs
// only the rows.  One 24 KB slot for both held 3 terms on average where a
// term's table is 5 KB (6 of 16 warps had a half term); apart, chunks have 5 to
// 8 terms: 3,001 shots of such a program 0.332 -> 0.248 ms, of the 40-output
// program 0.219 -> 0.191.
//
// What bounds it: issued instructions and their latency (four warps a
// scheduler, 54 % of the issue slots, the ALU pipe 47 % busy, shared memory
// 45 %, HBM idle).  Of ~5,100 warp instructions a term and 2,048 shots the
// rows take ~2,400, the values ~1,700, the draws ~900.
#pragma once
#include "sample_tile.cuh"
#include "slice.h"

namespace ksim {

// The ring: NSLOT slots of rows, one of tables, a barrier each.
constexpr int SLICE_RING = NSLOT * SLICE_SLOT + SLICE_TABLES;

// Shared memory of a sliced tile of `shots` (a power of two up to 2,048):
// parameter rows, result planes, then the barriers and the ring.
// (The rows of a 2,048-shot tile are two regions, 1,024 shots each.)
__host__ __device__ constexpr int slice_region(int rows) { return (rows + 1) * SLICE_ROW; }
__host__ __device__ constexpr int slice_rows_bytes(int rows, int shots)
{
    return slice_region(rows) * (shots > 1024 ? 2 : 1);
}
__host__ __device__ constexpr int slice_ring_off(int rows, int planes, int shots)
{
    return (slice_rows_bytes(rows, shots) + planes * shots + 127) & ~127;
}
__host__ __device__ constexpr int slice_smem_bytes(int rows, int planes, int shots)
{
    return slice_ring_off(rows, planes, shots) + BAR_BYTES + SLICE_RING;
}

// Two CTAs of a shape fit an SM (228 KB, 1 KB of a CTA reserved).
__host__ __device__ constexpr bool slice_two_ctas(int rows, int planes, int shots)
{
    return 2 * (slice_smem_bytes(rows, planes, shots) + 1024) <= 228 * 1024;
}

// The most a sliced CTA takes (254 parameters, 2,048 shots): every sliced
// kernel's dynamic shared-memory bound, whatever a launch asks for, so
// launches from several threads do not lower it for one another.
constexpr int SLICE_SMEM_MAX = slice_smem_bytes(SLICE_MAX_ROWS, SLICE_MAX_PLANES, 2048);
static_assert(SLICE_SMEM_MAX <= 226 * 1024, "shared memory of a CTA");

struct W2 {
    uint32_t a, b;
};
__device__ __forceinline__ W2 operator^(W2 x, W2 y) { return {x.a ^ y.a, x.b ^ y.b}; }
__device__ __forceinline__ W2 operator&(W2 x, W2 y) { return {x.a & y.a, x.b & y.b}; }
__device__ __forceinline__ W2 operator|(W2 x, W2 y) { return {x.a | y.a, x.b | y.b}; }
__device__ __forceinline__ W2 operator~(W2 x) { return {~x.a, ~x.b}; }
__device__ __forceinline__ W2 maj(W2 x, W2 y, W2 z)
{
    return {(x.a & y.a) | (x.a & z.a) | (y.a & z.a), (x.b & y.b) | (x.b & z.b) | (y.b & z.b)};
}

// The four rows of a group for this lane's 64 shots.  lane8: the shared
// address of the lane's column of the parameter rows.  A slot's address is one
// dot product (byte k of the word times the row pitch, plus the column); slots
// beyond a row's parameters name the zero row.  ONE: the warp has one lane
// group, so its lanes take the same path, and the common lengths have one
// each; else the lanes of several groups run two slots at a time together.
__device__ __forceinline__ W2 slice_ld(uint32_t x, int k, uint32_t lane8)
{
    W2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.a), "=r"(v.b)
                 : "r"(__dp4a(x, (uint32_t)SLICE_ROW << (8 * k), lane8)));
    return v;
}
__device__ __forceinline__ void slice_two(const uint4 &u, int k, uint32_t lane8, W2 (&r)[SLICE_GROUP])
{
    const uint32_t v[4] = {u.x, u.y, u.z, u.w};
    W2 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = slice_ld(v[i], k, lane8);
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = slice_ld(v[i], k + 1, lane8);
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = r[i] ^ x[i] ^ y[i];
}
__device__ __forceinline__ void slice_rows(uint32_t entry, const uint8_t *chunk, uint32_t lane8, W2 (&r)[SLICE_GROUP])
{
    const uint4 *p = (const uint4 *)(chunk + 16u * (entry & 0xFFFFu));
    int n = (int)((entry >> 16) & 0xFFu);
    const uint4 inv = p[0], u = p[1];
    r[0] = {inv.x, inv.x};
    r[1] = {inv.y, inv.y};
    r[2] = {inv.z, inv.z};
    r[3] = {inv.w, inv.w};
    slice_two(u, 0, lane8, r);
    if (n <= 2) return;
    slice_two(u, 2, lane8, r);
    for (n -= 4, p += 2; n > 0; n -= 4, ++p) {
        const uint4 v = *p;
        slice_two(v, 0, lane8, r);
        if (n <= 2) break;
        slice_two(v, 2, lane8, r);
    }
}

__device__ __forceinline__ W2 slice_shfl(W2 x, int o)
{
    return {__shfl_xor_sync(~0u, x.a, o), __shfl_xor_sync(~0u, x.b, o)};
}

// Add the counters (planes FROM..TO - 1) of lane groups o lanes apart.
template <int FROM, int TO, int N>
__device__ __forceinline__ void slice_add(W2 (&c)[N], int o)
{
    W2 carry = {0u, 0u};
#pragma unroll
    for (int i = FROM; i < TO; ++i) {
        const W2 x = slice_shfl(c[i], o), t = maj(c[i], x, carry);
        c[i] = c[i] ^ x ^ carry;
        carry = t;
    }
}

// 4 x 4 byte transpose: byte k of word i to byte i of word k.
__device__ __forceinline__ void transpose4(uint32_t (&x)[4])
{
    const uint32_t a0 = __byte_perm(x[0], x[1], 0x5140), a1 = __byte_perm(x[0], x[1], 0x7362);
    const uint32_t b0 = __byte_perm(x[2], x[3], 0x5140), b1 = __byte_perm(x[2], x[3], 0x7362);
    x[0] = __byte_perm(a0, b0, 0x5410);
    x[1] = __byte_perm(a0, b0, 0x7632);
    x[2] = __byte_perm(a1, b1, 0x5410);
    x[3] = __byte_perm(a1, b1, 0x7632);
}

// Eight planes of 32 shots to 32 bytes: word r, byte j of q holds bit 8 j + r
// of every plane, plane k in its bit k.  Stored as the 32 bytes at o.
__device__ __forceinline__ void slice_store(uint32_t (&p)[8], uint8_t *o)
{
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) {
        const uint32_t m = d == 4 ? 0x0F0F0F0Fu : d == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i & d) continue;
            const uint32_t x = p[i], y = p[i + d];
            p[i] = (x & m) | ((y << d) & ~m);
            p[i + d] = ((x >> d) & m) | (y & ~m);
        }
    }
    ((uint4 *)o)[0] = make_uint4(p[0], p[1], p[2], p[3]);
    ((uint4 *)o)[1] = make_uint4(p[4], p[5], p[6], p[7]);
}

// The warp's place in a rows pass: L lanes a group, this lane's group and its
// column.  The result words li and li + L are stored by the first two groups,
// or both by the only one.
struct SliceLane {
    int L, li, grp, n_grp;
    uint32_t lane8;
};
template <bool ONE, typename F>
__device__ __forceinline__ void slice_finish(const SliceLane &ln, F &&store)
{
    if (ONE) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) store(h, ln.li + 32 * h);
    } else if (ln.grp < 2) {
        store(ln.grp, ln.li + ln.grp * ln.L);
    }
}
__device__ __forceinline__ uint32_t slice_pick(W2 x, int h) { return h ? x.b : x.a; }

// x += b0 + ... + b3 in planes of weight 1, 2 (carries of weight 4 returned).
__device__ __forceinline__ W2 slice_add4(W2 &x0, W2 &x1, W2 b0, W2 b1, W2 b2, W2 b3)
{
    const W2 t0 = maj(x0, b0, b1);
    x0 = x0 ^ b0 ^ b1;
    const W2 t1 = maj(x0, b2, b3);
    x0 = x0 ^ b2 ^ b3;
    const W2 f = maj(x1, t0, t1);
    x1 = x1 ^ t0 ^ t1;
    return f;
}
// The same into one plane, the carries xored into the next.
__device__ __forceinline__ void slice_add4x(W2 &x0, W2 &x1, W2 b0, W2 b1, W2 b2, W2 b3)
{
    const W2 t0 = maj(x0, b0, b1);
    x0 = x0 ^ b0 ^ b1;
    const W2 t1 = maj(x0, b2, b3);
    x0 = x0 ^ b2 ^ b3;
    x1 = x1 ^ t0 ^ t1;
}

// The X half of a term: planes 0-6 X + 1 (0: dead), 7 S, the parity of X's
// count after its class-1 rows.  The halves are loops of their own, X's without
// a look at the role: of ~3,200 warp instructions a term's rows pass took for
// 2,048 shots, ~700 were the one loop's role dispatch and ~450 register moves
// (606,208 shots of the 40-output program: 0.783 -> 0.711 ms).
template <bool ONE>
__device__ __forceinline__ void slice_x(const uint8_t *chunk, const SliceTerm &d, uint8_t *planes, int plane_bytes,
                                        const SliceLane &ln)
{
    const uint32_t *list = (const uint32_t *)(chunk + 16 * (int)d.list_off16) + (int)d.n_k;
    const int n_x = d.n_x1 + d.n_x0, n = n_x + d.n_xp, n_x1 = d.n_x1, step = ONE ? 1 : ln.n_grp;
    const uint32_t one = ONE || ln.grp == 0 ? ~0u : 0u;
    W2 a[7], kill = {0u, 0u}, s = {one, one};
    a[0] = {one, one};
#pragma unroll
    for (int i = 1; i < 7; ++i) a[i] = {0u, 0u};
    int q = ONE ? 0 : ln.grp;
    for (; q < n_x; q += step) {
        W2 r[SLICE_GROUP];
        slice_rows(list[q], chunk, ln.lane8, r);
        W2 c = slice_add4(a[0], a[1], r[0], r[1], r[2], r[3]);
#pragma unroll
        for (int i = 2; i < 7; ++i) {
            const W2 t = a[i] & c;
            a[i] = a[i] ^ c;
            c = t;
        }
        if (q < n_x1) s = a[0];  // the parity so far, complemented by `one`
    }
    s = {s.a ^ one, s.b ^ one};
    for (; q < n; q += step) {
        const uint32_t e = list[q];
        W2 r[SLICE_GROUP];
        slice_rows(e, chunk, ln.lane8, r);
        if (e >> 24 == SQ_PPX) {
            s = s ^ (r[0] & r[1]);
            s = s ^ (r[2] & r[3]);
        } else {
            kill = kill | r[0] | r[1];
            kill = kill | r[2] | r[3];
        }
    }
    for (int o = ONE ? 32 : ln.L; o < 32; o <<= 1) {
        s = s ^ slice_shfl(s, o);
        kill = kill | slice_shfl(kill, o);
        slice_add<0, 7>(a, o);
    }
    uint8_t *out = planes + (int)d.plane * plane_bytes;
    slice_finish<ONE>(ln, [&](int h, int word) {
        uint32_t p[8];
        const uint32_t live = ~slice_pick(kill, h);
#pragma unroll
        for (int i = 0; i < 7; ++i) p[i] = slice_pick(a[i], h) & live;
        p[7] = slice_pick(s, h);
        slice_store(p, out + 32 * word);
    });
}

// The K half: planes a[0..2] K, y[] and z[] the p and q counts.
template <bool ONE>
__device__ __forceinline__ void slice_k(const uint8_t *chunk, const SliceTerm &d, uint8_t *planes, int plane_bytes,
                                        const SliceLane &ln)
{
    const uint32_t *list = (const uint32_t *)(chunk + 16 * (int)d.list_off16);
    const int n = d.n_k;
    W2 a[3], y[4], z[4];
#pragma unroll
    for (int i = 0; i < 3; ++i) a[i] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = z[i] = {0u, 0u};
    bool n9 = false;
    for (int q = ONE ? 0 : ln.grp; q < n; q += ONE ? 1 : ln.n_grp) {
        const uint32_t e = list[q], role = e >> 24;
        W2 r[SLICE_GROUP];
        slice_rows(e, chunk, ln.lane8, r);
        if (role == SQ_PPK) {
            a[2] = a[2] ^ (r[0] & r[1]);
            a[2] = a[2] ^ (r[2] & r[3]);
        } else if (role == SQ_W1) {
            a[2] = a[2] ^ slice_add4(a[0], a[1], r[0], r[1], r[2], r[3]);
        } else if (role == SQ_W2) {
            slice_add4x(a[1], a[2], r[0], r[1], r[2], r[3]);
        } else if (role == SQ_W4) {
            a[2] = a[2] ^ r[0] ^ r[1];
            a[2] = a[2] ^ r[2] ^ r[3];
        } else {  // SQ_N9
            n9 = true;
#pragma unroll
            for (int i = 0; i < SLICE_GROUP; i += 2) {
                W2 yb = ~(r[i] | r[i + 1]), zb = r[i] & r[i + 1];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const W2 ty = y[b] & yb, tz = z[b] & zb;
                    y[b] = y[b] ^ yb;
                    z[b] = z[b] ^ zb;
                    yb = ty;
                    zb = tz;
                }
            }
        }
    }
    n9 = __any_sync(~0u, n9);
    for (int o = ONE ? 32 : ln.L; o < 32; o <<= 1) {
        slice_add<0, 3>(a, o);
        if (n9) {
            slice_add<0, 4>(y, o);
            slice_add<0, 4>(z, o);
        }
    }
    uint8_t *out = planes + ((int)d.plane + 1) * plane_bytes;
    const bool even = d.flags & ST_EVEN, wide = d.flags & ST_WIDE;
    slice_finish<ONE>(ln, [&](int h, int word) {
        const uint32_t k0 = slice_pick(a[0], h), k1 = slice_pick(a[1], h), k2 = slice_pick(a[2], h);
        const uint32_t y0 = slice_pick(y[0], h), y1 = slice_pick(y[1], h), y2 = slice_pick(y[2], h),
                       z0 = slice_pick(z[0], h), z1 = slice_pick(z[1], h), z2 = slice_pick(z[2], h);
        if (wide) {
            uint32_t w[8] = {y0, y1, y2, slice_pick(y[3], h), z0, z1, z2, slice_pick(z[3], h)};
            slice_store(w, out + plane_bytes + 32 * word);
        }
        // class e (e + 1) / 2 + z, e = y + z <= 4 (ST_WIDE: 0)
        const uint32_t on = wide ? 0u : ~0u;
        const uint32_t e0 = y0 ^ z0, c0 = y0 & z0, e1 = y1 ^ z1 ^ c0;
        const uint32_t e2 = (y2 | z2 | (y1 & z1) | (y1 & c0) | (z1 & c0)) & on;
        const uint32_t t0 = (e0 ^ e1) & on, t1 = (e1 | e2) & on, t2 = e0 & e1 & on;  // e (e + 1) / 2; its bit 3 is e2
        const uint32_t w0 = z0 & on, w1 = z1 & on, w2 = z2 & on;
        const uint32_t q0 = t0 & w0, q1 = (t1 & w1) | (t1 & q0) | (w1 & q0), q2 = (t2 & w2) | (t2 & q1) | (w2 & q1);
        const uint32_t cl0 = t0 ^ w0, cl1 = t1 ^ w1 ^ q0, cl2 = t2 ^ w2 ^ q1, cl3 = e2 ^ q2;
        uint32_t p[8];
        p[0] = k1;
        p[1] = even ? cl0 : k0;
        p[2] = even ? cl1 : cl0;
        p[3] = even ? cl2 : cl1;
        p[4] = even ? cl3 : cl2;
        p[5] = even ? 0u : cl3;
        p[6] = 0u;
        p[7] = k2;
        slice_store(p, out + 32 * word);
    });
}

// u < rn(mag / prev), the draw of kokkos_sim.cpp:226-227, without the division
// where the product u * prev is clear of mag: t = rn(u prev) is within 2^-53
// of it relatively (normal t), so outside t (1 +- 2^-50) the quotient's
// rounding cannot change the comparison.  Everything else (and NaN, zeros,
// infinities beside infinities) divides.  flags: KSIM_FLAG_* raised.
static __device__ __noinline__ double slice_philox(uint64_t seed, uint64_t shot, uint32_t output)
{
    return philox_uniform(seed, shot, output);
}
static __device__ __noinline__ uint32_t slice_draw_exact(double u, double mag, double prev)
{
    const double ratio = __ddiv_rn(mag, prev);
    return (u < ratio ? 1u : 0u) | (!(prev > 0.0) ? (uint32_t)KSIM_FLAG_PREV_NONPOSITIVE << 8 : 0u) |
           (ratio != ratio ? (uint32_t)KSIM_FLAG_NAN << 8 : 0u);
}
__device__ __forceinline__ bool slice_draw(double u, double mag, double prev, uint32_t &flags)
{
    const double t = dmul(u, prev);
    bool bit = mag > dmul(t, 1.0 + 0x1p-50);
    if (!(t > 0x1p-900) || !(bit || mag < dmul(t, 1.0 - 0x1p-50))) {
        const uint32_t x = slice_draw_exact(u, mag, prev);
        bit = x & 1u;
        flags |= x >> 8;
    }
    return bit;
}

// xorshift_uniform with the 53-bit integer converted through two exact
// doubles (2^84 + hi 2^32, 2^52 + lo) instead of a 64-bit conversion.
__device__ __forceinline__ double slice_xorshift(uint64_t &s)
{
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    const uint64_t v = s >> 11;
    const double h = __hiloint2double(0x45300000, (int)(uint32_t)(v >> 32));
    const double l = __hiloint2double(0x43300000, (int)(uint32_t)v);
    return dmul(dadd(dsub(h, 0x1p84), dsub(l, 0x1p52)), 0x1p-53);
}

__device__ __forceinline__ uint32_t byte_of(uint32_t x, int k) { return (x >> (8 * k)) & 0xFFu; }

// A thread's bytes of a result plane.
template <int N>
__device__ __forceinline__ uint32_t slice_plane(uint32_t p)
{
    uint32_t x;
    if (N == 4) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(p));
    else asm volatile("ld.shared.u8 %0, [%1];" : "=r"(x) : "r"(p));
    return x;
}

// Issue the copies of a chunk's rows and of its tables (`bytes` at `off` of
// the job's stream) as the gidx-th of the CTA.
__device__ __forceinline__ void slice_issue(const SampleJob &j, int64_t off, uint32_t bytes, uint32_t gidx,
                                            uint64_t *bar, uint8_t *slots)
{
    const int slot = (int)(gidx & (NSLOT - 1));
    mbar_arrive_expect_tx(&bar[slot], bytes);
    tma_bulk_g2s(slots + (size_t)slot * SLICE_SLOT, j.image + off, bytes, &bar[slot]);
}
__device__ __forceinline__ void slice_issue_tables(const SampleJob &j, int64_t off, uint32_t bytes, uint64_t *bar,
                                                   uint8_t *slots)
{
    mbar_arrive_expect_tx(&bar[NSLOT], bytes);
    tma_bulk_g2s(slots + NSLOT * SLICE_SLOT, j.image + off, bytes, &bar[NSLOT]);
}
// A chunk's wait, the same for all lanes: usually the copy is there; what
// follows a first try that ran out is out of line (a job's own bound counts
// every poll).
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}
static __device__ __noinline__ bool slice_wait_out(uint64_t *bar, uint32_t parity, long long polls)
{
    return polls > 0 ? mbar_poll(bar, parity, polls) : mbar_wait(bar, parity);
}
__device__ __forceinline__ bool slice_wait(const SampleJob &j, uint64_t *bar, uint32_t parity)
{
    return __all_sync(~0u, (j.wait_limit <= 0 && mbar_try(bar, parity)) ||
                               slice_wait_out(bar, parity, j.wait_limit));
}
// The ring's barriers (once per CTA).
__device__ __forceinline__ void slice_ring_init(uint64_t *bar)
{
    if (threadIdx.x == 0) mbar_init(&bar[NSLOT], 1);
    ring_init(bar);
}

__device__ __forceinline__ uint2 lds64(uint32_t a)
{
    uint2 x;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x.x), "=r"(x.y) : "r"(a));
    return x;
}

// Sample shots [s0, s_end) of job j in a tile of `shots`, S of them a thread
// (slice_tile_ok; threads past shots / S only share the rows pass).  smem: the
// CTA's shared memory, parameter rows first, planes at planes_off.  Returns
// false after a wait timeout (the CTA must then stop using the ring).
// EVAL: instead of sampling, the job's chunks are one graph's and its rows are
// whole parameter vectors; |A| (EVAL_ABS) or A (EVAL_COMPLEX) goes to j.amp, or,
// after a wait timeout, SLICE_UNWRITTEN to the tile's first row.
template <int S, bool CG = false, int EVAL = -1>
__device__ __forceinline__ bool slice_tile(const SampleJob &j, const int64_t s0, const int64_t s_end, int shots,
                                           uint8_t *smem, int planes_off, uint64_t *bar, uint32_t &g)
{
    uint8_t *slots = (uint8_t *)bar + BAR_BYTES;
    static_assert(S == 1 || S == 4 || S == 8, "shots per thread");
    const int tid = threadIdx.x, lane = tid & 31, nthr = (int)blockDim.x;
    uint8_t *planes = smem + planes_off;
    const int plane_bytes = shots;
    const int F = j.F, R = j.s_rows;
    const int region = slice_region(R);
    constexpr bool ONE = S == 8;  // (S = 8 comes with 2,048 shots)
    const int warp = __shfl_sync(~0u, tid >> 5, 0);  // (the same in all lanes, also to the compiler)
    SliceLane ln;
    ln.L = ONE ? 32 : shots >> 6;
    ln.li = lane & (ln.L - 1);
    ln.grp = lane / ln.L;
    ln.n_grp = 32 / ln.L;
    ln.lane8 = smem_u32(smem) + 8u * (uint32_t)(ln.li & 15) + (uint32_t)((ln.li >> 4) * region);
    // this thread's shots: bits sh_bit(0), ... of word w (32 shots)
    //   S = 8: bits r + 8 k and r + 4 + 8 k;  S = 4: bits r + 8 k;  S = 1: bit r
    const bool mine = tid * S < shots;
    const int w = tid * S >> 5, r = S == 8 ? tid & 3 : S == 4 ? tid & 7 : lane;
    const int64_t sh0 = s0 + 32 * w + r;
    auto sh_of = [&](int k) { return sh0 + (S == 8 ? 8 * (k & 3) + 4 * (k >> 2) : 8 * k); };
    // its bytes of a result plane: word r of the 32 (and r + 4), or one byte
    const int byte0 = S == 1 ? 32 * w + 4 * (lane & 7) + (lane >> 3) : 32 * w + 4 * r;
    uint32_t act = 0;
#pragma unroll
    for (int k = 0; k < S; ++k) act |= mine && sh_of(k) < s_end ? 1u << k : 0u;
    const bool warp_any = __any_sync(~0u, act != 0);
    // word w of a parameter row: lane w mod L's 64-bit column
    const int wl = w & (ln.L - 1);
    const int wcol = (wl & 15) * 8 + (wl >> 4) * region + (w >= ln.L ? 4 : 0);
    auto put_row = [&](int row, const bool (&x)[S]) {
        uint32_t b[S];
#pragma unroll
        for (int k = 0; k < S; ++k) b[k] = __ballot_sync(~0u, x[k]);
        uint8_t *o = smem + row * SLICE_ROW + wcol;
        if (S == 8) {  // byte r of the word: the word's nibble of ballots r and r + 4
            const uint32_t lo = r & 2 ? (r & 1 ? b[3 % S] : b[2 % S]) : (r & 1 ? b[1 % S] : b[0]);
            const uint32_t hi = r & 2 ? (r & 1 ? b[7 % S] : b[6 % S]) : (r & 1 ? b[5 % S] : b[4 % S]);
            const int sh = 4 * (w & 7);
            if (mine) o[r] = (uint8_t)(((lo >> sh) & 15u) | ((hi >> sh) & 15u) << 4);
        } else if (S == 4) {  // byte w & 3 of each ballot
            const uint32_t sel = (uint32_t)(w & 3) | ((uint32_t)(4 + (w & 3)) << 4);
            const uint32_t x0 = __byte_perm(b[0], b[1 % S], sel), x1 = __byte_perm(b[2 % S], b[3 % S], sel);
            if (mine && r == 0) *(uint32_t *)o = __byte_perm(x0, x1, 0x5410);
        } else {
            if (mine && r == 0) *(uint32_t *)o = b[0];
        }
    };

    // Parameter rows p .. p + 3 (those below F) from each shot's four bytes.  S =
    // 4, 8: byte transposes give each thread a parameter's bits of four shots in
    // the low bits of four bytes; shifted to their places they are combined over
    // the word's lanes, each of the first four ending up with one parameter.
    auto put_rows4 = [&](int p, uint32_t (&x)[S]) {
        if (S == 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t word = __ballot_sync(~0u, x[0] & (1u << (8 * i)));
                if (mine && r == 0 && p + i < F) *(uint32_t *)(smem + (p + i) * SLICE_ROW + wcol) = word;
            }
        } else {
            uint32_t t[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int h = 0; h < S / 4; ++h) {
                uint32_t y[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) y[k] = x[(4 * h + k) % S] & 0x01010101u;
                transpose4(y);
#pragma unroll
                for (int i = 0; i < 4; ++i) t[i] |= y[i] << (r + 4 * h);
            }
            const bool o1 = r & 1, o2 = r & 2;
            const uint32_t s0 = o1 ? t[0] : t[2], s1 = o1 ? t[1] : t[3];
            uint32_t u0 = o1 ? t[2] : t[0], u1 = o1 ? t[3] : t[1];
            u0 |= __shfl_xor_sync(~0u, s0, 1);
            u1 |= __shfl_xor_sync(~0u, s1, 1);
            uint32_t v = o2 ? u1 : u0;
            v |= __shfl_xor_sync(~0u, o2 ? u0 : u1, 2);
            if (S == 4) v |= __shfl_xor_sync(~0u, v, 4);
            const int row = p + 2 * (r & 1) + ((r >> 1) & 1);
            if (mine && r < 4 && row < F) *(uint32_t *)(smem + row * SLICE_ROW + wcol) = v;
        }
    };

    // parameter rows: the f bits (16 or 4 bytes of a row at a time where rows
    // allow it), outputs zero for graph 0, the zero row
    int p0 = 0;
    if (!j.f_sel && ((((uintptr_t)j.f) | (uintptr_t)j.f_stride) & 15u) == 0) {
        for (; p0 + 16 <= F; p0 += 16) {
            uint4 x[S];
#pragma unroll
            for (int k = 0; k < S; ++k)
                x[k] = ((act >> k) & 1u) ? ldj<CG>((const uint4 *)(j.f + sh_of(k) * j.f_stride + p0))
                                         : make_uint4(0u, 0u, 0u, 0u);
            uint32_t y[S];
#define KSIM_ROWS4(M, Q)                                       \
    _Pragma("unroll") for (int k = 0; k < S; ++k) y[k] = x[k].M; \
    put_rows4(p0 + 4 * Q, y);
            KSIM_ROWS4(x, 0) KSIM_ROWS4(y, 1) KSIM_ROWS4(z, 2) KSIM_ROWS4(w, 3)
#undef KSIM_ROWS4
        }
    }
    if (!j.f_sel && ((((uintptr_t)j.f) | (uintptr_t)j.f_stride) & 3u) == 0) {
        for (; p0 + 4 <= F; p0 += 4) {
            uint32_t x[S];
#pragma unroll
            for (int k = 0; k < S; ++k)
                x[k] = ((act >> k) & 1u) ? ldj<CG>((const uint32_t *)(j.f + sh_of(k) * j.f_stride + p0)) : 0u;
            put_rows4(p0, x);
        }
    }
    for (; p0 < F; p0 += 4) {
        uint32_t x[S] = {};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = min(p0 + i, F - 1);
            const int col = j.f_sel ? ldj<CG>(j.f_sel + p) : p;
#pragma unroll
            for (int k = 0; k < S; ++k)
                if ((act >> k) & 1u) x[k] |= (uint32_t)ldj<CG>(j.f + sh_of(k) * j.f_stride + col) << (8 * i);
        }
        put_rows4(p0, x);
    }
    auto fill_rows = [&](int from, int to, uint32_t x) {
        for (int i = tid; i < (to - from) * (SLICE_ROW / 4); i += nthr) {
            ((uint32_t *)(smem + from * SLICE_ROW))[i] = x;
            if (ln.L > 16) ((uint32_t *)(smem + region + from * SLICE_ROW))[i] = x;
        }
    };
    fill_rows(F, R + 1, 0u);

    uint64_t rng[S];
    double prev[S], sre[S], sim[S];
#pragma unroll
    for (int k = 0; k < S; ++k) {
        rng[k] = xorshift_init(j.seed, (uint64_t)(j.shot_offset + sh_of(k)));
        prev[k] = 0.0;
        sre[k] = 0.0;
        sim[k] = 0.0;
    }
    uint32_t flags = 0, idle_flags = 0;  // (idle: shots past the job's end)
    const int nch = j.n_chunks;
    __syncthreads();
    if (tid == 0)
        for (int c = 0; c < NSLOT && c < nch; ++c) {
            const ChunkDir d = ld_chunk<CG>(j.cdir + c);
            slice_issue(j, d.off, (uint32_t)d.bytes, g + (uint32_t)c, bar, slots);
            if (c == 0) slice_issue_tables(j, d.off + d.bytes, (uint32_t)d.pad0, bar, slots);
        }

    for (int c = 0; c < nch; ++c) {
        const uint32_t gc = g + (uint32_t)c, par = (gc / NSLOT) & 1u;
        const int slot = (int)(gc & (NSLOT - 1));
        const uint8_t *chunk = slots + (size_t)slot * SLICE_SLOT;
        const SliceTerm *terms = (const SliceTerm *)(chunk + SLICE_HEAD);
        const bool ok = slice_wait(j, &bar[slot], par);
        const SliceChunk &d = *(const SliceChunk *)chunk;
        const int nt = ok ? d.n_terms : 0;

        // rows pass: one half term a warp
        for (int task = warp; task < 2 * nt; task += nthr >> 5)
            if (task < nt) slice_k<ONE>(chunk, terms[task], planes, plane_bytes, ln);
            else slice_x<ONE>(chunk, terms[task - nt], planes, plane_bytes, ln);
        if (__syncthreads_or(!slice_wait(j, &bar[NSLOT], gc & 1u) || !ok)) {
            if (tid == 0) {
                atomicOr(j.status, (uint32_t)KSIM_FLAG_WAIT_TIMEOUT);
                if (EVAL >= 0) ((uint64_t *)j.amp)[(EVAL == EVAL_ABS ? 1 : 2) * s0] = SLICE_UNWRITTEN;
                mbar_wait(&bar[slot], par);
                mbar_wait(&bar[NSLOT], gc & 1u);
                if (c + 1 < nch) mbar_wait(&bar[slot ^ 1], ((gc + 1) / NSLOT) & 1u);
            }
            return false;
        }

        // values pass
        const uint8_t *tables = slots + NSLOT * SLICE_SLOT;
        // (addresses that the compiler is not to compute again for each term)
        uint32_t tb = smem_u32(tables), pb = smem_u32(planes) + (uint32_t)byte0;
        asm volatile("" : "+r"(tb), "+r"(pb));
        if (warp_any) {
            for (int t = 0; t < nt; ++t) {
                uint4 T;
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(T.x), "=r"(T.y), "=r"(T.z), "=r"(T.w)
                             : "r"(tb + (uint32_t)sizeof(SliceValue) * (uint32_t)t));
                const uint32_t fl = T.y >> 16, xs = T.y & 0xFFFFu, tw = T.x;
                const uint32_t pl0 = pb + (T.z >> 16) * (uint32_t)plane_bytes;
                const bool big = __any_sync(~0u, (fl & ST_BIG) != 0), wide = __any_sync(~0u, (fl & ST_WIDE) != 0);
                const uint32_t base = big ? 0u : tb + tw;
                constexpr int N = S == 1 ? 1 : 4;
#pragma unroll
                for (int h = 0; h < (S == 8 ? 2 : 1); ++h) {
                    const uint32_t pl = pl0 + 16 * h;
                    const uint32_t xw = slice_plane<N>(pl), kw = slice_plane<N>(pl + plane_bytes);
                    const uint32_t xm = xw & 0x7F7F7F7Fu, km = kw & 0x7F7F7F7Fu;
                    uint32_t at[N];
#pragma unroll
                    for (int k = 0; k < N; ++k) at[k] = __dp4a(km, 8u << (8 * k), byte_of(xm, k) * xs + base);
                    if (wide) {
                        const uint32_t cw = slice_plane<N>(pl + 2 * plane_bytes);
                        const uint8_t *lut = tables + 16 * (int)(T.z & 0xFFFFu);
                        const uint32_t cs = (fl & ST_EVEN) ? 16u : 32u;
#pragma unroll
                        for (int k = 0; k < N; ++k) at[k] += (uint32_t)lut[byte_of(cw, k)] * cs;
                    }
                    // K's bit 1 has swapped the halves of the entry
                    uint2 a[N], b[N];
                    if (big) {
#pragma unroll
                        for (int k = 0; k < N; ++k) {
                            const uint8_t *p = j.image + 16 * (size_t)tw + at[k];
                            const uint8_t *q = (const uint8_t *)((uintptr_t)p ^ 8u);
                            a[k] = CG ? __ldcg((const uint2 *)p) : __ldg((const uint2 *)p);
                            b[k] = CG ? __ldcg((const uint2 *)q) : __ldg((const uint2 *)q);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < N; ++k) {
                            a[k] = lds64(at[k]);
                            b[k] = lds64(at[k] ^ 8u);
                        }
                    }
                    // times i^(K1 + 2 (K2 ^ S)): the signs go to bit 63
                    const uint32_t sI = xw ^ kw, sR = sI ^ (kw << 7);
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const uint32_t ra = (sR << (24 - 8 * k)) & 0x80000000u, ib = (sI << (24 - 8 * k)) & 0x80000000u;
                        double &re = sre[4 * h + k], &im = sim[4 * h + k];
                        re = dadd(re, __hiloint2double((int)(a[k].y ^ ra), (int)a[k].x));
                        im = dadd(im, __hiloint2double((int)(b[k].y ^ ib), (int)b[k].x));
                    }
                }
            }
        }

        if (EVAL >= 0) {
            if (d.end_of_graph) {
#pragma unroll
                for (int q = 0; q < S; ++q) {
                    if (!((act >> q) & 1u)) continue;
                    if (EVAL == EVAL_ABS) {
                        j.amp[sh_of(q)] = dsqrt(dadd(dmul(sre[q], sre[q]), dmul(sim[q], sim[q])));
                    } else {
                        j.amp[2 * sh_of(q)] = sre[q];
                        j.amp[2 * sh_of(q) + 1] = sim[q];
                    }
                }
            }
        } else if (d.end_of_graph) {
            const int k = d.graph;
            bool bit[S] = {};
            if (warp_any) {
#pragma unroll
                for (int q = 0; q < S; ++q) {
                    const double mag = dsqrt(dadd(dmul(sre[q], sre[q]), dmul(sim[q], sim[q])));
                    sre[q] = 0.0;
                    sim[q] = 0.0;
                    const int64_t sh = sh_of(q);
                    if (j.amp && ((act >> q) & 1u)) j.amp[sh * (int64_t)(j.n_out + 1) + k] = mag;
                    if (k == 0) {
                        prev[q] = mag;
                    } else {
                        const double u = j.rng_mode == KSIM_RNG_PHILOX
                                             ? slice_philox(j.seed, (uint64_t)(j.shot_offset + sh), (uint32_t)(k - 1))
                                             : slice_xorshift(rng[q]);
                        bit[q] = slice_draw(u, mag, prev[q], ((act >> q) & 1u) ? flags : idle_flags);
                        prev[q] = bit[q] ? mag : dsub(prev[q], mag);
                    }
                }
            }
            if (k == 0) {  // from graph 1 on, outputs not yet sampled are the trying bit
                fill_rows(F, R, ~0u);
            } else {
                put_row(F + k - 1, bit);
            }
        }
        const int64_t ahead_off = 16 * (int64_t)d.ahead_off16, tab_off = 16 * (int64_t)d.tab_off16;
        const uint32_t ahead_bytes = d.ahead_bytes, tab_bytes = d.tab_bytes;
        __syncthreads();
        if (tid == 0 && c + 1 < nch) {
            slice_issue_tables(j, tab_off, tab_bytes, bar, slots);
            if (c + NSLOT < nch) slice_issue(j, ahead_off, ahead_bytes, gc + NSLOT, bar, slots);
        }
    }
    g += (uint32_t)nch;
    if (EVAL >= 0) return true;

    // output rows, eight or four columns at once where they are contiguous and
    // aligned
    if (mine) {
        auto word_of = [&](int i) { return *(const uint32_t *)(smem + (F + i) * SLICE_ROW + wcol) >> r; };
        const uintptr_t place = j.out_cols ? 1u : (uintptr_t)(j.out + j.out_col0) | (uintptr_t)j.out_stride;
        int i = 0;
        if (S > 1 && (place & 3u) == 0) {
            uint8_t *out = j.out + j.out_col0;
            const bool pairs = (place & 7u) == 0;
            while (i + 4 <= j.n_out) {
                const bool two = pairs && i + 8 <= j.n_out;
                uint32_t x[2][4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    x[0][k] = word_of(i + k);
                    x[1][k] = two ? word_of(i + 4 + k) : 0u;
                }
#pragma unroll
                for (int h = 0; h < (S + 3) / 4; ++h) {
                    uint32_t y[2][4];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) y[q][k] = (x[q][k] >> (4 * h)) & 0x01010101u;
                        transpose4(y[q]);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int sh = (4 * h + k) % S;
                        if (!((act >> sh) & 1u)) continue;
                        uint8_t *o = out + sh_of(sh) * j.out_stride + i;
                        if (two) *(uint2 *)o = make_uint2(y[0][k], y[1][k]);
                        else *(uint32_t *)o = y[0][k];
                    }
                }
                i += two ? 8 : 4;
            }
        }
        for (; i < j.n_out; ++i) {
            const uint32_t x = word_of(i);
            const int64_t col = j.out_cols ? (int64_t)ldj<CG>(j.out_cols + i) : j.out_col0 + i;
#pragma unroll
            for (int k = 0; k < S; ++k)
                if ((act >> k) & 1u)
                    j.out[sh_of(k) * j.out_stride + col] =
                        (uint8_t)((x >> (S == 8 ? 8 * (k & 3) + 4 * (k >> 2) : 8 * k)) & 1u);
        }
    }
    if (flags) atomicOr(j.status, flags);
    return true;
}

}  // namespace ksim
