// The 70 dot products of a heavy ghost's WENO extrapolation (bc1.rs:221-244)
// with its stencil data d (rows of S_0..S_4 and w_{r,k}): how the rows lie in
// the ghost's record, and the row layout of d that keeps the loads of different
// orders in different shared-memory banks. Used by the ghost update
// (ghosts.cu), its vector-Jacobian product (adjoint.cu) and the packing of
// the records (context.cu).
//
// The rows of order r are S_r's (r+1)^2 rows, then w_{r,0..r}. The ghost update
// gives a ghost 16 lanes, four rows of one order (a quad) each: lanes 0-6 and 15
// order 4 (lane 15 its last two rows), 7-11 order 3, 12-14 order 2; quad_row
// orders a quad's rows so that the rows of D which the lanes touch together lie
// in different shared-memory banks. Term by term a quad is stored as two
// 16-byte chunks of two rows; at term b the lanes' first chunks lie side by
// side, then their second ones, so each load of a half-warp is one contiguous
// run: terms 0-8 hold 16 + 15 chunks (all lanes), 9-15 13 + 12 (orders 4, 3),
// 16-24 8 + 7 (order 4). Orders 1 (3 pairs x 4 terms) and 0 (1 pair) follow.
#pragma once

namespace rh3t {

constexpr int GR_SEG1 = 9 * 31, GR_SEG2 = GR_SEG1 + 7 * 25, GR_ORDER1 = GR_SEG2 + 9 * 15;
constexpr int GR_ORDER0 = GR_ORDER1 + 12, GR_CHUNKS = GR_ORDER0 + 1; // 602 chunks of 16 bytes

// row i (0-3) of a quad: rotated by quad / 2, so that D rows 4 quad + (i + quad
// / 2) mod 4 of eight consecutive quads differ mod 8 (the last quad of order 4
// holds two rows, both in its first chunk)
__host__ __device__ constexpr int quad_row(int r, int quad, int i) {
    return 4 * quad + ((i + (r == 4 && quad == 7 ? 0 : quad >> 1)) & 3);
}
// chunk h (0, 1) of a quad of order 2, 3 or 4 at term b
__host__ __device__ __forceinline__ int quad_chunk(int r, int quad, int h, int b) {
    const int lane = r == 4 ? (quad < 7 ? quad : 15) : (r == 3 ? 7 + quad : 12 + quad);
    if (b < 9) return 31 * b + (h ? 16 + lane : lane);
    if (b < 16) return GR_SEG1 + 25 * (b - 9) + (h ? 13 + lane : (lane == 15 ? 12 : lane));
    return GR_SEG2 + 15 * (b - 16) + (h ? 8 + lane : (lane == 15 ? 7 : lane));
}
// place of term b of row R of order r in the record's rows
__host__ __device__ __forceinline__ int row_place(int r, int R, int b) {
    if (r == 0) return 2 * GR_ORDER0 + R;
    if (r == 1) return 2 * (GR_ORDER1 + 3 * b + (R >> 1)) + (R & 1);
    const int quad = R >> 2, i = ((R & 3) - (r == 4 && quad == 7 ? 0 : quad >> 1)) & 3;
    return 2 * quad_chunk(r, quad, i >> 1, b) + (i & 1);
}

// Row of D holding stencil node a of order r: the order blocks start at
// kDOff[r], whose residues mod 8 differ, so the 16-byte loads of D rows of
// different orders at the same position fall in different banks.
static __constant__ int kDOff[5] = {0, 1, 5, 14, 31};
__host__ __device__ constexpr int d_row(int a) { return a + (a >= 30 ? 1 : 0); }

// Schedule of the 70 dot products of the vector-Jacobian product, all six
// fields at once, as the 35 chunks' pairs of rows, in two slots a warp runs one
// after the other (25 and 4 terms at most): order << 8 | quad << 4 | chunk (orders
// 1 and 0: the pair for the quad); kPairNone = none
constexpr unsigned kPairNone = 0xffffffffu;
__host__ __device__ constexpr unsigned pair(int r, int quad, int h) { return (unsigned)(r << 8 | quad << 4 | h); }
static __constant__ unsigned kSlotA[32] = {  // orders 4 (lanes 0-14), 3 (15-24), 2 (25-30), 1 (31)
    pair(4, 0, 0), pair(4, 0, 1), pair(4, 1, 0), pair(4, 1, 1), pair(4, 2, 0), pair(4, 2, 1), pair(4, 3, 0),
    pair(4, 3, 1), pair(4, 4, 0), pair(4, 4, 1), pair(4, 5, 0), pair(4, 5, 1), pair(4, 6, 0), pair(4, 6, 1),
    pair(4, 7, 0),
    pair(3, 0, 0), pair(3, 0, 1), pair(3, 1, 0), pair(3, 1, 1), pair(3, 2, 0), pair(3, 2, 1), pair(3, 3, 0),
    pair(3, 3, 1), pair(3, 4, 0), pair(3, 4, 1),
    pair(2, 0, 0), pair(2, 0, 1), pair(2, 1, 0), pair(2, 1, 1), pair(2, 2, 0), pair(2, 2, 1), pair(1, 0, 0)};
static __constant__ unsigned kSlotB[32] = {  // the rest of order 1, order 0
    pair(1, 1, 0), pair(1, 2, 0), pair(0, 0, 0),
    kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone,
    kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone,
    kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone, kPairNone,
    kPairNone, kPairNone};

// the six fields of one row of d (rows are 48 bytes, 16-byte aligned)
__device__ __forceinline__ void load_d6(const double* p, double d[6]) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = q[0], b = q[1], c = q[2];
    d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y; d[4] = c.x; d[5] = c.y;
}

__device__ __forceinline__ void store_d6(double* p, const double d[6]) {
    double2* q = reinterpret_cast<double2*>(p);
    q[0] = make_double2(d[0], d[1]);
    q[1] = make_double2(d[2], d[3]);
    q[2] = make_double2(d[4], d[5]);
}

} // namespace rh3t
