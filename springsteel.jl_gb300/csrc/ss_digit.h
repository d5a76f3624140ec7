// ss_digit.h — ring DFTs as tensor-core products of digit slices
// (ss_digit.cu): plan, device tables and launches.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <memory>
#include <utility>
#include <vector>

#include "ss_internal.h"

struct ss_grid;

namespace ss {

struct DigitTables;

// Digit formats.  A binary64 column scaled into (-1, 1) is 54-bit fixed point (a
// matrix entry 53-bit): a leading digit of at most 512 (256) and five balanced
// base-512 digits; a binary32 one is 28-bit fixed point, a leading base-256 and
// two base-1024 digits.  Every digit is an integer of at most 512 and exact in
// binary16.
template <typename T>
struct DigitFormat;
template <>
struct DigitFormat<double> {
    static constexpr int kDigits = 6;
    static constexpr int kSums = 7;     // accumulators D_s = Σ_{i+j=s} y_i x_j, s = 0..6
    static constexpr int kCols = 32;    // data columns of one accumulator half
    static constexpr int kChunk = 6;    // K-steps of 16 per accumulator drain
    static constexpr int kStages = 6;
    static constexpr int kVars = 5;     // ring outputs as columns: f, ∂λ, ∂λλ, ∂r, ∂rr
};
template <>
struct DigitFormat<float> {
    static constexpr int kDigits = 3;
    static constexpr int kSums = 3;
    static constexpr int kCols = 80;
    static constexpr int kChunk = 12;
    static constexpr int kStages = 8;
    static constexpr int kVars = 4;     // ∂λ, ∂λλ, ∂r, ∂rr; f keeps the binary32 FFT's rounding
};
constexpr int kDigitRows = 128;                       // matrix rows of one tile (TMEM lanes)
constexpr int kDigitPlane = kDigitRows * 16 * 2;      // bytes of one digit plane of a K-step
template <typename T>
SS_HD constexpr int digit_a_bytes() { return DigitFormat<T>::kDigits * kDigitPlane; }
template <typename T>
SS_HD constexpr int digit_half_bytes() { return DigitFormat<T>::kDigits * DigitFormat<T>::kCols * 32; }
template <typename T>
SS_HD constexpr int digit_b_bytes() { return 2 * digit_half_bytes<T>(); }

constexpr int kDigitVariants = 5;   // f, ∂λ, ∂λλ, ∂r, ∂rr; a format's columns are the last kVars
constexpr int kDigitGroup = 8;      // items whose columns are interleaved
constexpr int kNanColumn = 0x7fffffff;  // column exponent of a column that holds an infinity or NaN
// Headroom of the binary64 inverse sums.  A term of a ring point is below 2^53 (2^54 of
// data × 2^53 of matrix, over 2^54) in its cosine and its sine part, so a point of a ring
// of n = ri + 1 is below √2·n·2^53 (1.27·n·2^53 is reached where all re = ± im), which
// passes 2^63 at n = 725.  Rings above that keep their quadrant parts (each below
// (n/2 + 1)·2^53 < 2^63) halved, at an exponent one higher: good for n ≤ 1448.  The
// forward sums (at most n terms below 2^53 in one part) fit for n ≤ 1023.
constexpr int kDigitFullRing = 724;
constexpr int kDigitMaxRing = 1023;
constexpr int kDigitMaxRingF32 = 2047;

// One ring of n = ri + 1 (L = 4n points) seen by the digit kernels.  The points
// λ_l = 2π(l + (ri − 1)/2)/L are p = (l + shift) mod L on the grid θ_p = 2π(p + half/2)/L,
// half = 1 for odd n, which is symmetric about 0 and π/2: a quadrant m = 0..n−1
// (n odd) or 0..n (n even) of four parts,
//   Ce = Σ_{k even} a_k cos kθ_m, Co (k odd), Se = −Σ_{k even} b_k sin kθ_m, So,
// gives x(θ) = Ce + Co + Se + So and its reflections.  Rows of part q kept in
// memory: m = lo[q]..lo[q] + cnt[q] − 1 at off[q] (the others are zero); 4n in all.
struct DigitRing {
    int n, half, shift, kmax;
    int te, to;            // K-steps of the even and odd parts
    int rt;                // row tiles of the quadrant
    int cnt[4], lo[4], off[4];
    int L;
    int64_t jofs, fofs;
    int64_t cosofs;        // cos(2πt/8n), t = 0..2n, in the quarter-wave table
    int64_t a_tile;        // first A tile of the ring
    // forward: rows are the wavenumbers 2j + parity, K the quadrant positions
    int tm, rtf;           // K-steps, row tiles of a part
    int64_t af_tile;       // first A tile of the ring's forward matrices
    int64_t dofs;          // phase roundings δ_k, k = 1..ri, at [dofs + k − 1]
};
inline SS_HD int digit_steps(const DigitRing &r, int part) { return (part & 1) ? r.to : r.te; }
// tiles of the parts before `part`, `per` tiles per K-step
inline SS_HD int64_t digit_part_base(const DigitRing &r, int part, int64_t per) {
    return per * ((part > 0 ? r.te : 0) + (part > 1 ? r.to : 0) + (part > 2 ? r.te : 0));
}

// One tile product: 128 quadrant rows of one part × 2·kCols columns, T K-steps
struct DigitItem {
    int64_t a_tile, b_tile;
    int ring, part, row_tile, col_tile, steps, _pad;
};

// A group of rings whose B digits fit the scratch together: one split launch
// and one product launch
struct DigitSpan {
    int r0, r1;            // rings (0-based)
    int item0, items;
};
struct DigitSet {
    std::vector<DigitSpan> spans;
    const DigitItem *items = nullptr;
    const int64_t *btile = nullptr;  // per ring: first B tile within its span
};

// Column stages (binary64): matrix digits of M_0, M_1, M_2 per variable and the
// 32-position blocks of the quadrants
struct DigitColumns {
    bool on = false;
    int steps = 0, zblocks = 0, buffers = 1, raws = 1;
    const uint8_t *M = nullptr;
    const int *mexpo = nullptr;
    const int *weight = nullptr;           // mode exponents taken from the matrices' columns into the data
    const int2 *blocks = nullptr;
    std::vector<int> first;          // first block of every ring, their number at the end
    bool fon = false;                // forward (binary64): K-steps of levels, blocks of 32 modes, lanes of a column
    int fsteps = 0, fblocks = 0, fgroup = 4;
    const uint8_t *fM = nullptr;
    const int *fexpo = nullptr;
};

// Binary32 column stage: 16-position blocks of the quadrants (ring, first position) and
// the first block of every ring
struct QuadBlocks {
    const int2 *blocks = nullptr;
    std::vector<int> first;
};

struct DigitPlan {
    bool on = false;
    int col_tiles = 0, col_tiles_fwd = 0;
    const DigitRing *rings = nullptr;
    std::vector<DigitRing> ring_host;
    std::vector<int> cap_host;
    std::shared_ptr<DigitTables> tables;  // hold A and Af
    void *A = nullptr;      // digit planes of the inverse DFT matrices
    void *Af = nullptr;     // and of the forward ones
    const int *delta = nullptr;   // δ_k·2^70
    const int *cap = nullptr;     // per item: its variable's kmax
    void *H = nullptr;      // RL: quadrant parts
    void *B = nullptr;      // digit planes of one span's ring spectra
    int *expo = nullptr;    // [variant][item][ring] column exponents
    int *err = nullptr;     // host-mapped: a bounded wait gave up
    DigitSet whole, whole_fwd;
    std::vector<DigitSet> chunks, chunks_fwd;
    DigitColumns columns;
    QuadBlocks quads;       // binary32: the column stage reads the parts
};

// The device arrays of one plan in one allocation: host arrays are appended, then the plan's
// other buffers, and every pointer is set once the block is there (an allocation takes 35 µs, a
// copy 8; a small grid's plan had 17 of each)
struct DigitBlock {
    std::vector<unsigned char> host;
    size_t bytes = 0;
    std::vector<std::pair<void **, size_t>> at;
    size_t place(size_t n, size_t align = 256) {
        const size_t o = (bytes + align - 1) / align * align;
        bytes = o + std::max<size_t>(n, 16);
        return o;
    }
    template <typename V>
    void put(const V **dst, const std::vector<V> &src) {
        const size_t o = place(src.size() * sizeof(V));
        host.resize(bytes);
        if (!src.empty()) std::memcpy(host.data() + o, src.data(), src.size() * sizeof(V));
        at.push_back({(void **)dst, o});
    }
    void room(void **dst, size_t n) { at.push_back({dst, place(n, 1024)}); }
    bool build(std::vector<void *> &allocs) {
        void *p = nullptr;
        if (cudaMalloc(&p, bytes) != cudaSuccess) { cudaGetLastError(); return false; }
        allocs.push_back(p);
        for (const auto &q : at) *q.first = (char *)p + q.second;
        return cudaMemcpy(p, host.data(), host.size(), cudaMemcpyHostToDevice) == cudaSuccess;
    }
};

// Builds the plan of a grid (tables included); a grid the rule leaves to
// the FFT kernels, or whose tables do not fit the device, keeps on = false.
int32_t digit_build(ss_grid *g, const std::vector<RingDesc> &rings);
// ring_inverse of every ring (chunk < 0) or of one radial chunk: G → H
int32_t digit_ring_inverse(ss_grid *g, cudaStream_t st, int chunk, int *launches);
// ring_forward likewise: C → F
int32_t digit_ring_forward(ss_grid *g, cudaStream_t st, int chunk, int *launches);
// The rings of many FP64 RL grids in three launches: rings of the same length share one product,
// whose columns are the items of all grids that have it.  Bit for bit the single grids' results.
struct DigitJoined {
    const ss_grid *owner = nullptr;  // the grid of most rings, whose matrices serve
    const void *refs = nullptr;
    const int *count = nullptr;
    void *B = nullptr;
    int *expo = nullptr;
    int items = 0;
    const DigitItem *work[2] = {nullptr, nullptr};  // inverse, forward
    const int64_t *btile[2] = {nullptr, nullptr};
    int nwork[2] = {0, 0};
};
constexpr int kDigitJoinedLaunches = 3;
bool digit_joins(const ss_grid *g);  // an RL grid whose rings are one span
// sets of at most kDigitScratchBytes of digits; device memory goes to `mem`
int32_t digit_join_plan(std::vector<ss_grid *> gs, std::vector<void *> &mem, std::vector<DigitJoined> &out);
cudaError_t digit_join_launch(const DigitJoined &J, bool fwd, cudaStream_t st);
void digit_free(ss_grid *g);
// after a synchronisation: SS_DEVICE_TIMEOUT once if a bounded wait of the products gave up
int32_t digit_status(ss_grid *g);
int32_t digit_columns_build(ss_grid *g, const std::vector<ChebHost> &cheb);
// cheb_forward of the columns [col0, col1): physical slot 1 → C
int32_t digit_columns_forward(ss_grid *g, cudaStream_t st, int64_t col0, int64_t col1);
// cheb_inverse of the parts digit_ring_inverse left in H: H → physical
int32_t digit_columns_inverse(ss_grid *g, cudaStream_t st, int chunk);

}  // namespace ss
