// slice.h — the sliced term stream: a component's terms as sign counts and
// value tables, for the bit-sliced sampling kernel (slice_tile.cuh).
//
// Every factor of a term (zx_eval.hpp:101-165) is, up to a constant per
// column, a unit times powers of three elements:
//   NodePhases 1 + s w^j (s = +-1): w^(6 m) lambda^(m3 - m1) over the columns
//     with s = -1 (lambda = 1 + sqrt2), or 0 (j = 0, s = -1);
//   HalfPi, PiProducts: w^k;
//   PhasePairs 1 + w^a + w^b - w^(a+b), by the classes (a, b mod 4):
//     one of them 0     2 w^k;
//     both 2            (2 + 2i) w^k if the signs agree, else 0;
//     one 2, one odd    kappa lambda^x w^k, x = 1 iff the signs agree;
//     both odd          p w^k or q w^k (the primes above 3) if the signs
//                       agree (one for each sign), else (1 + i) w^k.
// So a term's value is w^K times a tabulated element selected by
//   X  the lambda exponent (plus a constant): a count of parity rows,
//   y, z  how many columns contributed p and q,
// and 0 if a kill row is set.  K (mod 8) is a sum of rows with weights 1, 2, 4
// and of products of row pairs with weight 4 (6 r = 6 + 2 (1 - r), 7 r = 7 +
// (1 - r) and 3 r = 7 r + 4 r mod 8 turn the other weights into these on the
// complemented row; the constants go into the tables, and so does w^(6X), so
// the NodePhases rows of classes 1 and 3 are counted once).  All of it is bit
// arithmetic on rows, which the kernel does for 64 shots per lane at once.
//
// The tables hold the term's finished complex doubles: the exact ring element
// (128-bit integers), cast and scaled with the reference's operations
// (zx_eval.hpp:166-178).  Halvings scale all four coefficients by a power of
// two, which commutes with every rounding while the scale stays a normal
// double, so the doubles are the reference's whatever its halving schedule.
// A component whose terms are all proven (the reference's int64 cannot wrap,
// scales normal), have finite approximation factors and fit the limits below
// gets a sliced stream; the others keep the term records (zring.cuh).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <vector>

#include "../../include/ksim_b200.h"
#include "image.h"

namespace ksim {

// Bytes between the parameter rows in shared memory: 1,024 shots.  Index
// slots are bytes, so at most 255 rows.
constexpr int SLICE_ROW = 128;
constexpr int SLICE_MAX_ROWS = 254;   // parameters; one more row is all zero
constexpr int SLICE_SLOT = 8192;      // bytes of a staged chunk's rows (two slots)
constexpr int SLICE_TABLES = 32768;   // bytes of its tables (one slot)
constexpr int SLICE_MAX_PLANES = 16;  // result bytes per shot of a chunk's terms
constexpr int SLICE_MAX_TERMS = 8;    // of a chunk
constexpr int SLICE_AHEAD = 2;        // chunks staged at once
// A stream's size is bounded: a term's table can take 550 KB (127 lambda steps,
// 136 classes) where its record takes 4, and building it grows alike (20,000
// terms of 15 p / q columns: 0.93 GB, 3.9 s, their records 83 MB, 0.9 s).  Up to
// the bound it pays: 200,000 shots of those take 31 ms, from the records 115.
constexpr size_t SLICE_MAX_BYTES = (size_t)1 << 30;

// Tile widths slice_tile takes: a power of two up to the rows' 1,024 shots, whole
// warps of S shots a lane (a lane without a shot of the tile would look up
// result bytes that nothing wrote) and no more threads than the CTA has; S = 8
// comes with two regions of rows.
constexpr bool slice_tile_ok(int S, int shots, int threads)
{
    return (shots & (shots - 1)) == 0 && shots >= 64 && shots >= 32 * S && shots <= S * threads &&
           (S == 8 ? shots == 2048 : shots <= 1024);
}

// In the first row of a tile whose evaluation gave up: a signalling NaN, which no
// arithmetic results in, so that the host learns of it from the results it copies
// anyway.  (Copying the status word back took 3.6 us of a 43 us call,
// a page-locked one 1.3 ms of a process's first.)
constexpr uint64_t SLICE_UNWRITTEN = 0x7FF0554E57524954ull;

// A chunk has two parts, staged by copies of their own: the rows (this head,
// its terms' SliceTerm, group lists and groups) and, behind them, the tables
// (SliceValue, then look-up tables and value tables).  The head says what a
// CTA needs to know of the chunk, of the next one's tables and of the rows of
// the chunk SLICE_AHEAD behind it.
struct SliceChunk {
    uint16_t n_terms, end_of_graph;
    uint32_t graph, ahead_bytes, ahead_off16, tab_bytes, tab_off16;
    uint32_t pad[2];
};
constexpr int SLICE_HEAD = sizeof(SliceChunk);
static_assert(SLICE_HEAD == 32, "SliceChunk layout");
constexpr int SLICE_BIG_TABLE = 16384;  // larger tables stay in global memory

enum : uint32_t { ST_WIDE = 1u, ST_BIG = 2u, ST_EVEN = 4u };

// A term's result per shot, one byte a plane:
//   X plane: X + 1, or 0 of a dead term (7 bits), bit 7 the parity S of the
//     class-1 rows;
//   K plane: bits 0-5 the table column in half entries (K's bit 1, then K's
//     bit 0 unless ST_EVEN, then the class of (y, z)), bit 7 K's bit 2
//     without S;
//   ST_WIDE (more than four p / q columns): a third plane y | z << 4, whose
//     class is read from a table of 256 (the K plane then has class 0).
// The value is table[X + 1][class][K0] * i^(2 (K2 ^ S) + K1), each entry a
// complex double (16 bytes); table[0] is zero.

// Roles of a term's rows, in stream order.  The K half: K by weight 1, 2, 4;
// p / q columns; weight-4 pairs.  The X half: X with and without S; weight-4
// pairs, into S; kill.
enum { SQ_W1, SQ_W2, SQ_W4, SQ_N9, SQ_PPK, SQ_X1, SQ_X0, SQ_PPX, SQ_KILL, SQ_ROLES };

// One term of a chunk, in either part.  Its rows come in groups of four, listed
// role by role as u32: bits 0-15 the group's offset in the chunk / 16, 16-23 its
// index slots a row, 24-27 the role.
constexpr int SLICE_GROUP = 4;
struct SliceTerm {
    uint16_t list_off16;  // group list (16-byte units, in the rows part)
    uint16_t plane;       // first result plane
    uint16_t flags;
    uint16_t n_k;         // groups of the K half
    uint16_t n_x1, n_x0;  // of X with and without S,
    uint16_t n_xp;        // of the X half's pairs and kill rows
    uint16_t pad;
};
static_assert(sizeof(SliceTerm) == 16, "SliceTerm layout");
struct SliceValue {
    uint32_t tab;        // byte offset of the table in the tables part (ST_BIG: / 16, in the image)
    uint16_t xs;         // table bytes per X step
    uint16_t flags;
    uint16_t lut_off16;  // ST_WIDE: 256 bytes, class of y | z << 4
    uint16_t plane;
    uint32_t pad;
};
static_assert(sizeof(SliceValue) == 16, "SliceValue layout");

struct SliceImage {
    bool ok = false;
    int rows = 0;        // parameter rows
    int max_planes = 0;  // of any chunk
    std::vector<uint8_t> bytes;
    std::vector<ChunkDir> chunks;  // off, bytes: the rows part; pad0: bytes of the tables behind it
};

// Build the sliced stream of a component whose image is `img` (build_image on
// the same descriptors).  out.ok is false when a term does not qualify or the
// stream would take more than max_bytes.
void build_slices(const ksim_graph_desc *gs, const HostImage &img, SliceImage &out,
                  size_t max_bytes = SLICE_MAX_BYTES);

}  // namespace ksim
