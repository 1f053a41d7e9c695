// Tiled production path of the fused step: a classify kernel and one compute kernel per list length.
//
// classify (tile_classify_kernel)
//   A block owns a (y, z) tile of TY x kTileZ voxels and marches along x over `xchunk` planes.  The 3x3x3
//   neighbourhoods come from a ring of three x-planes in shared memory (tile plus a one-voxel halo
//   in y and z; periodic wrap by index arithmetic).  The grains present in the three planes of the
//   window carry block-local slot numbers (at most kSlots, recycled as grains leave the window), and
//   every ring plane is held twice: per record its slots in entry order with a slot bitmask, and as
//   dense per-slot value planes dense[slot][plane][record] (zero where the grain is absent).  For
//   each voxel of the centre plane one thread
//     - derives the flag from its count and the "several fields" bits of the 27 records' words, and
//       copies bulk voxels to the output;
//     - discovers the candidate fields with bitmask operations, in the reference's order (own
//       fields, then new grains in stencil order and neighbour-list order);
//     - sums every field's Laplacian from the dense planes (27 loads and multiply-adds in stencil
//       order; the zero terms of absent neighbours leave every partial sum unchanged);
//     - writes the list to the work buffer and appends the voxel to its block's slice of the
//       bucket of its list length.
// compute (list_compute_kernel<N>)
//   One kernel per list length N = 2..kListCap over all the slices' entries of that length (a
//   small scan kernel turns the per-slice counts into offsets), split evenly over the CUDA blocks:
//   fully unrolled pair kinetics, driving force, projection, merge and finalize (the operation order
//   of list_step; from N = 5 on some of the arrays lie in local memory), new record written to the
//   output state.
// Lists longer than kListCap and voxels next to a grain without a window slot go to the general-path
// worklist, processed one warp per voxel (warp_step.cuh).
#pragma once
#include "step_kernel.cuh"
#include "warp_step.cuh"

namespace opgpu {

constexpr int kTileZ = kTileCols;
// distinct grains per 3-plane window: 16 for FP32 values, 14 for FP64 (its dense planes would
// otherwise leave room for only two blocks per SM)
template <class R>
struct WindowSlots {
    static constexpr int value = sizeof(R) == 8 ? 14 : 16;
};
constexpr int kSlotMap = 512;        // grain -> slot map entries
constexpr int kTileVolSlots = 512;      // grain-volume hash of the compute kernels
// Entries per record the plane loader keeps in registers.  FP32 has 96 registers at five blocks per SM
// and spills with six (256^3, classify: 1894 us with six, 1760 with four); FP64 has room for 160 at three
// blocks (it takes 135 to 144), and the records beyond four cost more (2060 with six, 2178 with four).
template <class R>
struct KeepEntries {
    static constexpr int value = sizeof(R) == 8 ? 6 : 4;
};
constexpr int kClassifyVolSlots = 128;  // grain-volume hash of the classify kernel (bulk voxels)
// Blocks of each per-length compute kernel: one per 4096 voxels of the grid, between 8 and 32 per
// SM (a finer split of each length's entries pays on large grids; on small ones the per-block
// set-up and flush of the grain-volume hash would cost more than it balances).
inline int compute_blocks(long long n)
{
    const long long b = n / 4096;
    return (int)(b < 148 * 8 ? 148 * 8 : (b > 148 * 32 ? 148 * 32 : b));
}
constexpr int kTileTY = kTileRows;   // tile rows (blocks of kTileZ x kTileRows threads)

template <int TY>
struct TileGeom {
    static constexpr int kRows = TY + 2;
    static constexpr int kCols = kTileZ + 2;
    static constexpr int kRecs = kRows * kCols;
    static constexpr int NT = kTileZ * TY;
};

// Flags of a record's word beside its slot bitmask.
constexpr uint32_t kWordSeveral = 0x80000000u;     // more than one field
constexpr uint32_t kWordUnslotted = 0x40000000u;   // a grain of the record has no slot

template <class R, int TY>
struct TileSmem {
    using Geo = TileGeom<TY>;
    static constexpr int kSlots = WindowSlots<R>::value;
    // per-slot values of the three ring planes (zero where absent).  Every slot's planes start at the
    // same bank, so that lanes reading different slots at neighbouring records do not conflict
    // (256^3, FP64: classify 2140 -> 2060 us).
    struct SlotPlanes {
        R at[3][Geo::kRecs];
        R pad[(128 - (3 * Geo::kRecs * sizeof(R)) % 128) % 128 / sizeof(R)];
    } dense[kSlots];
    double vol_sum[kClassifyVolSlots];
    uint2 slotl[3][Geo::kRecs];              // slot ids of the record in entry order, 4 bits each
    uint32_t word[3][Geo::kRecs];            // slot bitmask of the record | kWordSeveral | kWordUnslotted
    int vol_key[kClassifyVolSlots];
    alignas(16) int grain_of[16];            // slot -> grain (-1 = free or beyond kSlots)
    int lastpos[16];                         // last window position where the slot's grain occurs
    int pending[32];                         // grains of the incoming plane that need a slot
    unsigned nb[kListCap + 1];               // entries this block appended per list length
    unsigned woff;                           // bytes of work records this block wrote
    unsigned crowded;                        // voxels sent to the general path for a crowded window
    unsigned long long cnt[3];
    uint8_t map[kSlotMap];                   // hashed grain -> a slot that may hold it (check grain_of)
    uint8_t cntr[3][Geo::kRecs];             // entries per record
};

// Shared memory sets the resident blocks: five in FP32, three in FP64 (228 KB per SM, 1 KB of it
// reserved per block).
static_assert(sizeof(TileSmem<float, kTileTY>) <= 233472 / 5 - 1024, "FP32 classify: five blocks per SM");
static_assert(sizeof(TileSmem<double, kTileTY>) <= 233472 / 3 - 1024, "FP64 classify: three blocks per SM");

__device__ __forceinline__ unsigned slot_hash(int g) { return ((unsigned)g * 2654435761u) >> 23; }

// One term of the classify kernel's dense-plane Laplacian.  FP64: the reference's separate multiply
// and add (the FP64 unit is compiled without contraction).  FP32: one fused multiply-add, written
// out because the FP32 unit is compiled without contraction too (so that the adjoint can repeat its
// per-voxel arithmetic exactly); these Laplacians reach the forward and the adjoint alike through
// the work records, so their rounding only has to be the same in both, which it is.  Steps with
// anisotropic models or averaged driving forces (no adjoint) keep the separate operations of the
// generic kernel in either precision (FUSED = false).
template <bool FUSED>
__device__ __forceinline__ double lap_acc(double l, double w, double x) { return l + w * x; }
template <bool FUSED>
__device__ __forceinline__ float lap_acc(float l, float w, float x) { return FUSED ? __fmaf_rn(w, x, l) : l + w * x; }

// Slot of a grain in the window (-1 if the grain has none).  A window holds at most 16 grains, so
// the map hits but for a few per cent of the grains, whose entry another grain of the window took;
// they are searched for among the slots.
template <class S>
__device__ __forceinline__ int search_slot(const S& sm, int g)
{
    int k = -1;
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        const int4 four = reinterpret_cast<const int4*>(sm.grain_of)[q];
        if (four.x == g) k = 4 * q;
        if (four.y == g) k = 4 * q + 1;
        if (four.z == g) k = 4 * q + 2;
        if (four.w == g) k = 4 * q + 3;
    }
    return k;
}

template <class S>
__device__ __forceinline__ int find_slot(const S& sm, int g)
{
    const int k = sm.map[slot_hash(g)];
    return sm.grain_of[k] == g ? k : search_slot(sm, g);
}

// Records of a ring plane each thread handles.
template <int TY>
struct PlaneRegs {
    static constexpr int kPer = (TileGeom<TY>::kRecs + TileGeom<TY>::NT - 1) / TileGeom<TY>::NT;
};

// In-plane offset of record r (the same in every plane; -1 beyond the last record).
template <int TY>
__device__ __forceinline__ int record_offset(const StepParams& p, int r, int y0, int z0)
{
    using Geo = TileGeom<TY>;
    if (r >= Geo::kRecs) return -1;
    const int row = r / Geo::kCols, col = r - row * Geo::kCols;
    int yy = y0 - 1 + row; yy = yy < 0 ? yy + p.ny : (yy >= p.ny ? yy % p.ny : yy);
    int zz = z0 - 1 + col; zz = zz < 0 ? zz + p.nz : (zz >= p.nz ? zz % p.nz : zz);
    return yy * p.nz + zz;
}

// What a thread of the plane loader keeps from plane to plane: the in-plane offsets of its records
// and the next plane's counts (prefetched).
template <int TY>
struct PlaneState {
    int off[PlaneRegs<TY>::kPer];
    int cr[PlaneRegs<TY>::kPer];
};

// Counts of plane xp for this thread's records (issued one plane ahead of their use).
template <int TY>
__device__ __forceinline__ void prefetch_counts(const StepParams& p, const StepArrays& a, int xp, PlaneState<TY>& P)
{
    const uint8_t* __restrict__ cnt = a.cnt_in + (long long)xp * p.ny * p.nz;
#pragma unroll
    for (int i = 0; i < PlaneRegs<TY>::kPer; i++) P.cr[i] = P.off[i] >= 0 ? (int)cnt[P.off[i]] : 0;
}

// The loader state of a thread before its first plane xp.
template <int TY>
__device__ __forceinline__ void plane_begin(const StepParams& p, const StepArrays& a, int xp, int y0, int z0, int t,
                                            PlaneState<TY>& P)
{
#pragma unroll
    for (int i = 0; i < PlaneRegs<TY>::kPer; i++) P.off[i] = record_offset<TY>(p, t + i * TileGeom<TY>::NT, y0, z0);
    prefetch_counts<TY>(p, a, xp, P);
}

// Registers a thread keeps between the passes of the plane loader: the first KeepEntries entries of each
// of its records, the slots found so far (4 bits an entry, entries 0-7 and 8-15) and the entries
// without one.
template <class R, int TY>
struct PlaneLoad {
    int gr[PlaneRegs<TY>::kPer][KeepEntries<R>::value];
    R vr[PlaneRegs<TY>::kPer][KeepEntries<R>::value];
    uint32_t lst[PlaneRegs<TY>::kPer][2];
    uint32_t miss[PlaneRegs<TY>::kPer];
};

// Grain of entry s of record i (the kept ones without a dynamic register index).
template <class R, int TY>
__device__ __forceinline__ int kept_grain(const PlaneLoad<R, TY>& L, int i, int s, const int16_t* __restrict__ gin,
                                          long long N)
{
    int g = 0;
#pragma unroll
    for (int q = 0; q < KeepEntries<R>::value; q++)
        if (q == s) g = L.gr[i][q];
    return s >= KeepEntries<R>::value ? (int)gin[s * N] : g;
}

// Bringing plane xp (window position wpos) into ring slot `rs` -- slot lists, bitmask words and
// dense per-slot values; grains not yet in the window get a slot that no grain of the window uses --
// takes three passes with a barrier between each:
//   plane_scan    reads the records once (the first KeepEntries entries stay in registers) and finds their
//                 slots through the map; marks the slots as in use and collects the grains without
//                 one in `pending`; it touches only map and grain_of (read), lastpos and pending, so
//                 it may run while other threads still read the ring for the previous plane; returns
//                 whether this thread added a pending grain
//   plane_assign  warp 0 hands free slots to the pending grains (only needed when some thread
//                 added one)
//   plane_fill    slot lists, bitmask words and dense values of the incoming plane, clearing what
//                 the ring position held before and no longer holds
// P.cr holds the plane's counts on entry (prefetched) and the next plane's counts after plane_fill.
// Invariant of the dense planes: dense[k][rs][r] != 0 only if bit k of word[rs][r] is set.
template <class R, int TY>
__device__ __forceinline__ bool plane_scan(const StepParams& p, const StepArrays& a, TileSmem<R, TY>& S,
                                           int xp, int wpos, const PlaneState<TY>& P, PlaneLoad<R, TY>& L)
{
    using PR = PlaneRegs<TY>;
    const long long N = p.n;
    const long long base = (long long)xp * p.ny * p.nz;
    const int16_t* __restrict__ gin = a.idx_in + base;
    const R* __restrict__ vin = static_cast<const R*>(a.val_in) + base;
    bool added = false;
#pragma unroll
    for (int i = 0; i < PR::kPer; i++)
#pragma unroll
        for (int s = 0; s < KeepEntries<R>::value; s++)
            if (s < P.cr[i])
            {
                L.gr[i][s] = gin[s * N + P.off[i]];
                L.vr[i][s] = vin[s * N + P.off[i]];
            }
#pragma unroll
    for (int i = 0; i < PR::kPer; i++)
    {
        const int c = P.cr[i];
        uint32_t lst[2] = {0u, 0u};
        uint32_t miss = c > KeepEntries<R>::value ? ((1u << c) - 1u) & ~((1u << KeepEntries<R>::value) - 1u) : 0u;
#pragma unroll
        for (int s = 0; s < KeepEntries<R>::value; s++)
            if (s < c)
            {
                const int g = L.gr[i][s], k = S.map[slot_hash(g)];
                if (S.grain_of[k] == g)
                {
                    S.lastpos[k] = wpos;   // in use by the incoming plane: not free for plane_assign
                    lst[0] |= (uint32_t)k << (4 * s);
                }
                else miss |= 1u << s;
            }
        uint32_t left = 0;
        for (uint32_t m = miss; m; m &= m - 1u)
        {
            const int s = __ffs(m) - 1;
            const int g = kept_grain<R, TY>(L, i, s, gin + P.off[i], N);
            const int k = search_slot(S, g);
            if (k >= 0)
            {
                S.lastpos[k] = wpos;
                if (s < 8) lst[0] |= (uint32_t)k << (4 * s);
                else lst[1] |= (uint32_t)k << (4 * s - 32);
                continue;
            }
            added = true;
            left |= 1u << s;
            unsigned h = ((unsigned)g * 2654435761u) & 31u;
            for (int probe = 0; probe < 32; probe++)
            {
                const int q = atomicCAS(&S.pending[h], -1, g);
                if (q == -1 || q == g) break;
                h = (h + 1) & 31u;
            }
        }
        L.lst[i][0] = lst[0];
        L.lst[i][1] = lst[1];
        L.miss[i] = left;
    }
    return added;
}

template <class R, int TY>
__device__ __forceinline__ void plane_assign(TileSmem<R, TY>& S, int wpos, int t)
{
    // warp 0 hands free slots (grain gone from the window) to the pending grains
    if (t < 32)
    {
        const int g = S.pending[t];
        const bool valid = g >= 0;
        constexpr int kSlots = WindowSlots<R>::value;
        const bool is_free = t < kSlots && (S.grain_of[t & 15] < 0 || S.lastpos[t & 15] < wpos - 2);
        const unsigned fm = __ballot_sync(0xffffffffu, is_free);
        const unsigned vm = __ballot_sync(0xffffffffu, valid);
        const int rank = __popc(vm & ((1u << t) - 1u));
        // grains left without a slot are marked per record in plane_fill
        if (valid)
        {
            S.pending[t] = -1;
            if (rank < __popc(fm))
            {
                const int k = (int)__fns(fm, 0, rank + 1);
                S.grain_of[k] = g;
                S.lastpos[k] = wpos;
                S.map[slot_hash(g)] = (uint8_t)k;
            }
        }
    }
}

template <class R, int TY>
__device__ __forceinline__ void plane_fill(const StepParams& p, const StepArrays& a, TileSmem<R, TY>& S,
                                           int rs, int xp, int t, PlaneState<TY>& P, const PlaneLoad<R, TY>& L)
{
    using Geo = TileGeom<TY>;
    using PR = PlaneRegs<TY>;
    const long long N = p.n;
    const long long base = (long long)xp * p.ny * p.nz;
    const R* __restrict__ vin = static_cast<const R*>(a.val_in) + base;
#pragma unroll
    for (int i = 0; i < PR::kPer; i++)
    {
        const int r = t + i * Geo::NT;
        if (r >= Geo::kRecs) continue;
        const int c = P.cr[i];
        uint32_t lst[2] = {L.lst[i][0], L.lst[i][1]};
        // the slots plane_assign handed out
        uint32_t lost = 0;
        for (uint32_t m = L.miss[i]; m; m &= m - 1u)
        {
            const int s = __ffs(m) - 1;
            const int k = search_slot(S, kept_grain<R, TY>(L, i, s, a.idx_in + base + P.off[i], N));
            if (k < 0) lost |= 1u << s;
            else if (s < 8) lst[0] |= (uint32_t)k << (4 * s);
            else lst[1] |= (uint32_t)k << (4 * s - 32);
        }
        uint32_t msk = 0;
#pragma unroll
        for (int s = 0; s < KeepEntries<R>::value; s++)
            if (s < c && !((lost >> s) & 1u))
            {
                const int k = (int)(lst[0] >> (4 * s)) & 15;
                S.dense[k].at[rs][r] = L.vr[i][s];
                msk |= 1u << k;
            }
        for (int s = KeepEntries<R>::value; s < c; s++)
            if (!((lost >> s) & 1u))
            {
                const int k = (int)(lst[s >> 3] >> (4 * (s & 7))) & 15;
                S.dense[k].at[rs][r] = vin[s * N + P.off[i]];
                msk |= 1u << k;
            }
        for (uint32_t m = S.word[rs][r] & 0xFFFFu & ~msk; m; m &= m - 1u) S.dense[__ffs(m) - 1].at[rs][r] = R(0);
        S.word[rs][r] = msk | (c > 1 ? kWordSeveral : 0u) | (lost ? kWordUnslotted : 0u);
        S.slotl[rs][r] = make_uint2(lst[0], lst[1]);
        S.cntr[rs][r] = (uint8_t)c;
    }
    // counts of the next plane, for the next call
    prefetch_counts<TY>(p, a, xp == p.nx - 1 ? 0 : xp + 1, P);
}

// The three passes with their barriers, for kernels that do not overlap plane_scan with other work.
template <class R, int TY>
__device__ __forceinline__ void load_plane(const StepParams& p, const StepArrays& a, TileSmem<R, TY>& S,
                                           int rs, int xp, int wpos, int t, PlaneState<TY>& P)
{
    PlaneLoad<R, TY> L;
    plane_scan(p, a, S, xp, wpos, P, L);
    __syncthreads();
    plane_assign(S, wpos, t);
    __syncthreads();
    plane_fill(p, a, S, rs, xp, t, P, L);
}

// Offsets of the q-th Laplacian stencil element (LaplacianStencil::Set order): 27-point stencils
// enumerate x, y, z in -1..1; the 7-point stencil keeps the centre and the six faces.
template <int NS>
__device__ __forceinline__ constexpr int stencil_dx(int q) { return NS == 27 ? q / 9 - 1 : (q == 0 ? -1 : (q == 6 ? 1 : 0)); }
template <int NS>
__device__ __forceinline__ constexpr int stencil_dy(int q) { return NS == 27 ? (q / 3) % 3 - 1 : (q == 1 ? -1 : (q == 5 ? 1 : 0)); }
template <int NS>
__device__ __forceinline__ constexpr int stencil_dz(int q) { return NS == 27 ? q % 3 - 1 : (q == 2 ? -1 : (q == 4 ? 1 : 0)); }

// New grains of neighbour record (pl, r): append their slots (4 bits each) in the record's entry
// order.  n counts on past kListCap, ls then holds no list.
template <class R, int TY>
__device__ __forceinline__ void append_fresh(const TileSmem<R, TY>& S, int pl, int r, uint32_t fresh, uint32_t& ls, int& n)
{
    if ((fresh & (fresh - 1u)) == 0u)
    {
        // one new grain (the usual case): no order to look up
        ls |= (uint32_t)(__ffs(fresh) - 1) << ((4 * n) & 31);
        n++;
        return;
    }
    const int cu = S.cntr[pl][r];
    const uint2 list = S.slotl[pl][r];
    for (int s = 0; s < cu; s++)
    {
        const uint32_t k = ((s < 8 ? list.x : list.y) >> (4 * (s & 7))) & 15u;
        if ((fresh >> k) & 1u)
        {
            ls |= k << ((4 * n) & 31);
            n++;
        }
    }
}

template <class R, int TY, int NS, bool FUSED>
__global__ void __launch_bounds__(kTileZ * TY, sizeof(R) == 8 ? 3 : 5)
tile_classify_kernel(const __grid_constant__ StepParams p, const StepArrays a, int xchunk)
{
    using Geo = TileGeom<TY>;
    using Smem = TileSmem<R, TY>;
    constexpr int NT = Geo::NT;
    constexpr int kC = Geo::kCols;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);

    const int tz = threadIdx.x, ty = threadIdx.y, t = ty * kTileZ + tz;
    const int z0 = blockIdx.x * kTileZ, y0 = blockIdx.y * TY, x0 = blockIdx.z * xchunk;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const int x1 = min(x0 + xchunk, nx);
    const long long N = p.n;
    const long long plane = (long long)ny * nz;
    const int z = z0 + tz, y = y0 + ty;
    const bool inside = (z < nz) && (y < ny);
    const int blin = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    const long long nblocks = (long long)gridDim.x * gridDim.y * gridDim.z;
    const long long slice0 = (long long)blin * a.slice;
    unsigned char* __restrict__ wbase = a.wl + (long long)blin * a.wl_slice;
    R* __restrict__ vout = static_cast<R*>(a.val_out);

    for (int i = t; i < kClassifyVolSlots; i += NT) { S.vol_key[i] = -1; S.vol_sum[i] = 0.0; }
    for (int i = t; i < (int)(sizeof(S.dense) / sizeof(R)); i += NT) reinterpret_cast<R*>(S.dense)[i] = R(0);
    for (int i = t; i < 3 * Geo::kRecs; i += NT) (&S.word[0][0])[i] = 0u;
    if (t < 16) { S.grain_of[t] = -1; S.lastpos[t] = -1000; }
    for (int i = t; i < kSlotMap; i += NT) S.map[i] = 0;
    if (t < 32) S.pending[t] = -1;
    if (t <= kListCap) S.nb[t] = 0u;
    if (t < 3) S.cnt[t] = 0ull;
    if (t == 0) { S.woff = 0u; S.crowded = 0u; }
    unsigned wide = 0, ein = 0, eout = 0;
    uint32_t st = 0;
    int acc_g = -1;        // bulk-voxel volume accumulator of this thread
    double acc_v = 0.0;
    PlaneState<TY> P;
    plane_begin<TY>(p, a, x0 == 0 ? nx - 1 : x0 - 1, y0, z0, t, P);
    __syncthreads();

    const int rec0 = (ty + 1) * kC + (tz + 1);
    // words of the thread's column of records, kept while the block marches along x: per plane the
    // words of the three rows ORed over z (row0: the plane before the centre, row1: the centre plane,
    // row2: the plane after) and the middle word
    uint32_t row0[3], row1[3], row2[3], mid0 = 0, mid1 = 0, mid2 = 0;
#pragma unroll
    for (int dy = 0; dy < 3; dy++) row0[dy] = row1[dy] = row2[dy] = 0;

    // plane x0-1+j goes to ring slot j%3 at window position j-1; once three planes are in, the
    // centre plane x = x0+j-2 is processed (one call site of the plane loader keeps the code small)
    const int nj = (x1 - x0) + 2;
    for (int j = 0; j < nj; j++)
    {
        int xp = x0 - 1 + j;
        xp = xp < 0 ? xp + nx : (xp >= nx ? xp - nx : xp);
        // the scan of the incoming plane overlaps the other threads' work on the previous plane;
        // its barrier also ends that work, and the slot hand-out runs only when a grain is new
        {
            PlaneLoad<R, TY> L;
            const bool added = plane_scan(p, a, S, xp, j - 1, P, L);
            if (__syncthreads_or(added))
            {
                plane_assign(S, j - 1, t);
                __syncthreads();
            }
            plane_fill(p, a, S, j % 3, xp, t, P, L);
        }
        __syncthreads();
        mid0 = mid1; mid1 = mid2;
#pragma unroll
        for (int dy = 0; dy < 3; dy++)
        {
            row0[dy] = row1[dy];
            row1[dy] = row2[dy];
            const uint32_t* w = &S.word[j % 3][rec0 + (dy - 1) * kC];
            const uint32_t m = w[0];
            if (dy == 1) mid2 = m;
            row2[dy] = w[-1] | m | w[1];
        }
        if (j < 2 || !inside) continue;
        const int x = x0 + j - 2;
        const int sl0 = (j - 2) % 3, sl1 = (j - 1) % 3, sl2 = j % 3;
        const long long v = (long long)x * plane + (long long)y * nz + z;

        const int c = S.cntr[sl1][rec0];
        ein += c;
        // ---- flag and candidate discovery over the neighbours ------------------------------------
        // Candidates come in the reference's order: new grains of each neighbour in stencil order and
        // neighbour-list order.  The rows of three z-neighbours that hold a grain not seen in an
        // earlier row (nor in the voxel itself) are marked from the row words in registers; only
        // their records are visited (the others add nothing to the list).
        const uint32_t own = mid1 & 0xFFFFu;
        uint32_t multi = 0;
#pragma unroll
        for (int dy = 0; dy < 3; dy++) multi |= row0[dy] | row1[dy] | row2[dy];
        // a neighbour holding a grain the window has no slot for: the general path
        const bool window_bad = (multi & kWordUnslotted) != 0u;
        const int flag = c > 1 ? 2 : ((multi & kWordSeveral) ? 1 : 0);
        if (flag == 0)
        {
            // bulk voxel: carried over unchanged
            a.cnt_out[v] = (uint8_t)c;
            for (int s = 0; s < c; s++)
            {
                const int g = a.idx_in[s * N + v];
                const R phi = static_cast<const R*>(a.val_in)[s * N + v];
                a.idx_out[s * N + v] = (int16_t)g;
                vout[s * N + v] = phi;
                if (in_volume_window(p, v))
                {
                    // consecutive bulk voxels of a thread mostly belong to one grain: sum them in a
                    // register before the shared-memory add
                    if (g != acc_g)
                    {
                        if (acc_g >= 0) vol_insert_n(S.vol_key, S.vol_sum, kClassifyVolSlots, a.vol_acc, acc_g, acc_v);
                        acc_g = g;
                        acc_v = 0.0;
                    }
                    acc_v += (double)phi;
                }
            }
            eout += c;
            continue;
        }
        wide++;
        uint32_t ls = 0;
        int n = c;
        bool over = window_bad || c > kListCap;
        if (!over)
        {
            ls = S.slotl[sl1][rec0].x;   // c <= kListCap entries, unused nibbles are zero
            uint32_t seen = own;
            if (NS != 27)
            {
                // 7-point Laplacian: its neighbours first, then the gradient pass over all 26
                const uint32_t face[6] = {mid0, S.word[sl1][rec0 - kC], S.word[sl1][rec0 - 1],
                                          S.word[sl1][rec0 + 1], S.word[sl1][rec0 + kC], mid2};
#pragma unroll
                for (int q = 0; q < 6; q++)
                {
                    const uint32_t fresh = face[q] & 0xFFFFu & ~seen;
                    if (fresh)
                        append_fresh(S, q == 0 ? sl0 : (q == 5 ? sl2 : sl1),
                                     rec0 + (q == 1 ? -kC : (q == 2 ? -1 : (q == 3 ? 1 : (q == 4 ? kC : 0)))), fresh, ls, n);
                    seen |= fresh;
                }
            }
            if (NS == 27 || p.ng > 0)
            {
#pragma unroll
                for (int q = 0; q < 9; q++)
                {
                    const uint32_t w = q < 3 ? row0[q] : (q < 6 ? row1[q - 3] : row2[q - 6]);
                    const uint32_t fresh = w & 0xFFFFu & ~seen;
                    if (fresh == 0u) continue;
                    if ((fresh & (fresh - 1u)) == 0u)
                    {
                        ls |= (uint32_t)(__ffs(fresh) - 1) << ((4 * n) & 31);
                        n++;
                    }
                    else
                    {
                        // several in one row: in the order of its records
                        uint32_t left = fresh;
                        for (int dz = -1; dz <= 1; dz++)
                        {
                            const int pl = q < 3 ? sl0 : (q < 6 ? sl1 : sl2);
                            const int r = rec0 + (q - (q < 3 ? 1 : (q < 6 ? 4 : 7))) * kC + dz;
                            const uint32_t f = S.word[pl][r] & left;
                            if (f) append_fresh(S, pl, r, f, ls, n);
                            left &= ~f;
                        }
                    }
                    seen |= fresh;
                }
            }
            over = n > kListCap;
        }
        if (over || n < 2)
        {
            if (window_bad) atomicAdd(&S.crowded, 1u);
            const unsigned slot = atomicAdd(a.slow_count, 1u);
            if (slot < a.slow_cap) a.slow_list[slot] = (int)v;
            else st |= kStOverflowList;
            continue;
        }
        // ---- values and Laplacians from the dense planes into a work record ----------------------
        const int pad = ((2 * n + 7) / 8) * 8;
        const unsigned off = atomicAdd(&S.woff, (unsigned)(pad + 2 * n * (int)sizeof(R)));
        int16_t* rg = reinterpret_cast<int16_t*>(wbase + off);
        R* rv = reinterpret_cast<R*>(wbase + off + pad);
        for (int k = 0; k < n; k++)
        {
            const int s = (int)((ls >> (4 * k)) & 15u);
            R l = R(0);
#pragma unroll
            for (int q = 0; q < NS; q++)
            {
                const int dx = stencil_dx<NS>(q);
                const int pl = dx < 0 ? sl0 : (dx > 0 ? sl2 : sl1);
                const int r = rec0 + stencil_dy<NS>(q) * kC + stencil_dz<NS>(q);
                l = lap_acc<FUSED>(l, (R)p.lap_w[q], S.dense[s].at[pl][r]);
            }
            rg[k] = (int16_t)S.grain_of[s];
            rv[k] = S.dense[s].at[sl1][rec0];
            rv[n + k] = l;
        }
        const unsigned rank = atomicAdd(&S.nb[n], 1u);
        a.bucket[(long long)n * a.bucket_cap + slice0 + rank] =
            make_int2((int)v | (flag == 2 ? (int)0x80000000 : 0), (int)off);
    }
    __syncthreads();
    if (t >= 2 && t <= kListCap) a.bucket_count[t * nblocks + blin] = S.nb[t];
    if (t == 0 && S.crowded) atomicAdd(&a.counters[kCntCrowdedLast], (unsigned long long)S.crowded);
    if (acc_g >= 0) vol_insert_n(S.vol_key, S.vol_sum, kClassifyVolSlots, a.vol_acc, acc_g, acc_v);
    flush_block(a, wide, ein, eout, st, S.cnt, S.vol_key, S.vol_sum, kClassifyVolSlots, t, NT);
}

// Exclusive prefix of the per-slice bucket counts, one block per list length N = 2..kListCap:
// bucket_off[N][s] = entries of length N in slices before s, bucket_off[N][nslices] = their total.
static __global__ void __launch_bounds__(1024) bucket_scan_kernel(const StepArrays a, int nslices)
{
    __shared__ unsigned s_warp[32];
    const int N = blockIdx.x + 2;
    const unsigned* __restrict__ cnt = a.bucket_count + (long long)N * nslices;
    unsigned* __restrict__ off = a.bucket_off + (long long)N * (nslices + 1);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int per = (nslices + 1023) / 1024;
    const int s0 = min(t * per, nslices), s1 = min(s0 + per, nslices);
    unsigned sum = 0;
    for (int s = s0; s < s1; s++) sum += cnt[s];
    unsigned incl = sum;
    for (int o = 1; o < 32; o <<= 1)
    {
        const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0)
    {
        unsigned x = s_warp[lane];
        for (int o = 1; o < 32; o <<= 1)
        {
            const unsigned u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += u;
        }
        s_warp[lane] = x;   // inclusive over warps
    }
    __syncthreads();
    unsigned base = (w > 0 ? s_warp[w - 1] : 0u) + incl - sum;
    for (int s = s0; s < s1; s++) { off[s] = base; base += cnt[s]; }
    if (t == 0) off[nslices] = s_warp[31];
}

constexpr int kTogetherShare = 48;   // (see list_compute_kernel)
constexpr int kChunkTable = 128;   // 32-entry chunks of a compute block whose slices are tabulated
constexpr int kVolCache = 2;       // per-thread grain-volume cache of the compute kernels (four entries, of
                                   // which a thread's few voxels fill most once: FP32 step 4072 -> 4002 us)

// Stages 2-5 for lists of exactly N fields (compile-time), all arrays in registers; the operation
// order is that of list_step.  The entries of length N from all classify slices form one index
// range (bucket_off); each CUDA block takes an equal contiguous part of it, its warps 32
// consecutive entries at a time, so that no warp idles while another drains a long slice.
//
// Bound: issue and latency at 16-20 warps per SM -- FP64 arithmetic, pair-table loads and, for long
// lists, instruction fetch -- not bandwidth (N = 4 at 256^3: 0.41 ms for 0.09 ms of traffic).  Leaving
// out what repeats (one sum per field instead of one per pair and third field, one pass for merge and
// plausibility, no limits where no field leaves [0, 1]) took N = 2..8 at 256^3, FP64, from 235 443 519
// 396 283 185 147 us to 235 391 452 305 219 131 129 (233 389 412 281 206 126 117 with the block bounds and the
// smaller volume cache below).
//
// The kinetics have two branches, for lists whose grains all have their reference volume and for the
// others.  Each is a long straight line, fetched once by the warps that run it at about the same time;
// where small grains mix the two, warps in different branches fetch for themselves (128^3, mean grain
// 1728 voxels, FP32, N = 6: 13.5 of 22 cycles an instruction wait for it).  With `together` a block's
// warps take one branch in step: the general one if any list needs it, which gives a full list the same
// values.  N = 5, 6, 7, FP32: 227 400 338 -> 184 296 251 us, FP64: 228 364 208 -> 191 268 208; the step
// at 160^3 5.76 -> 4.89 and 7.98 -> 7.31 ms.  With grains of 8400 voxels the barrier costs a 256^3 step
// about 1 %, so that it goes by the share of the voxels on the general path (kTogetherShare: more than
// 3 % with grains of 1728 voxels, 0.2 % to 1.7 % with 3500, 0.2 % with 8400).
//
// N <= kListCap <= the stored fields per voxel, so a new record always fits.  AVG: averaged driving
// forces (a template parameter: the mask costs the plain step registers).
// Resident blocks: six for N <= 3, five for 4 and 5, three beyond (the registers each takes unbounded
// allow five, four and two to three): FP64 step at 256^3 4365 -> 4298 us.
template <class R, int N, bool AVG>
__global__ void __launch_bounds__(128, N <= 3 ? 6 : (N <= 5 ? 5 : 3)) list_compute_kernel(const __grid_constant__ StepParams p, const StepArrays a,
                                                           int nslices, bool together)
{
    constexpr int NP = N * (N - 1) / 2;
    __shared__ int s_key[kTileVolSlots];
    __shared__ double s_sum[kTileVolSlots];
    __shared__ unsigned long long s_cnt[3];
    __shared__ int s_chunk[kChunkTable];
    const int t = threadIdx.x;
    const unsigned* __restrict__ off = a.bucket_off + (long long)N * (nslices + 1);
    const unsigned total = off[nslices];
    // whole chunks of 32 entries for every warp of the block: a length with few entries then keeps
    // all warps of fewer blocks busy instead of one warp of many blocks (the others would wait at
    // the final barrier, holding their registers)
    const unsigned per = ((total + gridDim.x * blockDim.x - 1u) / (gridDim.x * blockDim.x)) * blockDim.x;
    const unsigned r0 = blockIdx.x * per;
    if (r0 >= total) return;
    const unsigned r1 = min(total, r0 + per);
    for (int i = t; i < kTileVolSlots; i += blockDim.x) { s_key[i] = -1; s_sum[i] = 0.0; }
    if (t < 3) s_cnt[t] = 0ull;
    // slice of each 32-entry chunk of the block's range
    const unsigned nchunks = (r1 - r0 + 31u) / 32u;
    const bool tabulated = nchunks <= (unsigned)kChunkTable;
    if (tabulated)
        for (unsigned c = t; c < nchunks; c += blockDim.x) s_chunk[c] = slice_of(off, nslices, r0 + 32u * c);
    __syncthreads();
    const long long N_ = p.n;
    const int2* __restrict__ buck = a.bucket + (long long)N * a.bucket_cap;
    // grain-volume contributions of this thread's voxels, most recent grain first (consecutive
    // voxels of a thread lie close together and mostly share their grains)
    int cg[kVolCache];
    double cv[kVolCache];
#pragma unroll
    for (int c = 0; c < kVolCache; c++) { cg[c] = -1; cv[c] = 0.0; }
    constexpr int kPad = ((2 * N + 7) / 8) * 8;
    R* __restrict__ vout = static_cast<R*>(a.val_out);
    uint32_t st = 0;
    unsigned eout = 0;
    for (unsigned first = r0; first < r1; first += blockDim.x)   // the same trip count for the block's warps
    {
        // (the lanes beyond the last entry repeat it and store nothing)
        const bool mine = first + t < r1;
        const unsigned e = mine ? first + t : r1 - 1u;
        // slice of the first entry of this one's chunk of 32, then its own
        int lo = tabulated ? s_chunk[(e - r0) >> 5] : slice_of(off, nslices, r0 + ((e - r0) & ~31u));
        while (off[lo + 1] <= e) lo++;   // off[nslices] = total > e
        const int2 ent = buck[(long long)lo * a.slice + (e - off[lo])];
        const unsigned char* __restrict__ wbase = a.wl + (long long)lo * a.wl_slice;
        const long long v = ent.x & 0x7fffffff;
        const int flag = (ent.x >> 31) ? 2 : 1;
        const int16_t* __restrict__ rg = reinterpret_cast<const int16_t*>(wbase + ent.y);
        const R* __restrict__ rv = reinterpret_cast<const R*>(wbase + ent.y + kPad);
        int g[N];
        R val[N], lap[N];
#pragma unroll
        for (int k = 0; k < N; k++)
        {
            g[k] = rg[k];
            val[k] = rv[k];
            lap[k] = rv[N + k];
        }
        // ---- pair kinetics ---------------------------------------------------------------------
        double vr[N];
        bool full = true;   // every grain at its reference volume (VolumeRatio 1)
#pragma unroll
        for (int k = 0; k < N; k++)
        {
            vr[k] = a.vr[g[k]];
            full = full && vr[k] == 1.0;
        }
        if (together) full = __syncthreads_and(full);
        R sg[NP];
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
            for (int j = i + 1; j < N; j++) sg[pair_pos(i, j, N)] = (R)pair_energy(p, a, g[i], g[j]);
        const R pref = (R)p.pref_do;
        double pv[NP];
        if (full && p.tj_factor == 0.0)
        {
            // The usual case.  With every scale 1 the factor h is one number (R(0.5) * (R(1) + R(1)) *
            // pref = pref), so lap + h*val is formed once per field instead of once per pair and third
            // field, the triple-junction term is absent and LocalN = N: the same operations on the
            // same operands as below, without their repetitions.
            const R norm_1 = (R)(1.0 / (double)N);
            R sum[N];
#pragma unroll
            for (int k = 0; k < N; k++) sum[k] = lap[k] + pref * val[k];
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int j = i + 1; j < N; j++)
                {
                    const int q = pair_pos(i, j, N);
                    R dphi = sg[q] * (sum[i] - sum[j]);
#pragma unroll
                    for (int k = 0; k < N; k++)
                    {
                        if (k == i || k == j) continue;
                        const R sbk = sg[j < k ? pair_pos(j, k, N) : pair_pos(k, j, N)];
                        const R sak = sg[i < k ? pair_pos(i, k, N) : pair_pos(k, i, N)];
                        dphi += (sbk - sak) * sum[k];
                    }
                    dphi *= (R)pair_mobility(p, a, g[i], g[j]) * norm_1;
                    pv[q] = (double)dphi;
                }
        }
        else
        {
            double localN;
            if (p.consider_nucleus_volume)
            {
                localN = 0.0;
#pragma unroll
                for (int k = 0; k < N; k++) localN += vr[k];
            }
            else
            {
                localN = (double)N;
            }
            const R norm_1 = (R)(1.0 / localN);
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int j = i + 1; j < N; j++)
                {
                    const int q = pair_pos(i, j, N);
                    const R scale = (vr[i] == 1.0 && vr[j] == 1.0) ? R(1) : (R)sqrt(vr[i] * vr[j]);
                    const R h = R(0.5) * (R(1) + scale) * pref;
                    R dphi = sg[q] * ((lap[i] + h * val[i]) - (lap[j] + h * val[j]));
                    if (N > 2)
                    {
#pragma unroll
                        for (int k = 0; k < N; k++)
                        {
                            if (k == i || k == j) continue;
                            const R sbk = sg[j < k ? pair_pos(j, k, N) : pair_pos(k, j, N)];
                            const R sak = sg[i < k ? pair_pos(i, k, N) : pair_pos(k, i, N)];
                            dphi += (sbk - sak) * (lap[k] + h * val[k]);
                            if (p.tj_factor != 0.0 || scale < R(1))
                            {
                                const int pA = a.gphase[g[i]], pB = a.gphase[g[j]], pG = a.gphase[g[k]];
                                const int P = p.nphases;
                                const R tj = (R)dmax_ref(p.tj_factor, (double)(R(1) - scale));
                                dphi += tj * pref
                                      * (((R)p.sigma_p[pA * P + pB] + (R)p.sigma_p[pB * P + pG]) + (R)p.sigma_p[pA * P + pG])
                                      * (val[i] * val[k] - val[j] * val[k]);
                            }
                        }
                    }
                    dphi *= (R)pair_mobility(p, a, g[i], g[j]) * norm_1 * scale;
                    pv[q] = (double)dphi;
                }
        }
        // ---- driving force (interface voxels only) ----------------------------------------------
        if (p.use_dg && flag == 2)
        {
            // stored fields are positive: the pairs of two of them are the ones averaging decides on
            unsigned reached = 0;
            if constexpr (AVG) reached = a.avg_mask[v];
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int j = i + 1; j < N; j++)
                {
                    double locdG;
                    if constexpr (AVG)
                        locdG = val[j] != R(0) && !((reached >> avg_bit(i, j)) & 1u) ? no_force(p, a, g[i], g[j])
                                                                                    : limited_force(p, a, g[i], g[j]);
                    else
                        locdG = limited_force(p, a, g[i], g[j]);
                    double norm = sqrt((double)val[i] * (double)val[j]);
                    if (a.gstage[g[i]] == 1 || a.gstage[g[j]] == 1) norm += 1.0e-6;
                    const double dpsi = locdG * (double)(R)pair_mobility(p, a, g[i], g[j]) * norm * p.pref_df;
                    pv[pair_pos(i, j, N)] += dpsi;
                }
        }
        // ---- projection ---------------------------------------------------------------------------
        const double dt = p.dt;
        bool any = false;   // lists of more than two fields: some increment is left
        if (NP == 1)
        {
            const double valueA = pv[0] * dt;
            const double old_value = (double)val[0];
            if ((old_value == 0.0 && valueA < 0.0) || (old_value == 1.0 && valueA > 0.0))
            {
                pv[0] = 0.0;
            }
            else
            {
                const double new_value = old_value + valueA;
                double norm = 1.0;
                if (new_value < 0.0) norm *= -old_value / valueA;
                else if (new_value > 1.0) norm *= (1.0 - old_value) / valueA;
                if (norm > DBL_EPSILON) pv[0] *= norm;
                else pv[0] = 0.0;
            }
        }
        else
        {
#pragma unroll
            for (int i = 0; i < N; i++)
            {
                if (val[i] != R(0) && val[i] != R(1)) continue;   // the sum is read at a bound only
                double dpsi = 0.0;
#pragma unroll
                for (int j = 0; j < N; j++)
                {
                    if (j == i) continue;
                    dpsi += (i < j) ? pv[pair_pos(i, j, N)] : pv[pair_pos(j, i, N)] * (-1.0);
                }
                if ((val[i] == R(0) && dpsi < 0.0) || (val[i] == R(1) && dpsi > 0.0))
                {
#pragma unroll
                    for (int j = 0; j < N; j++)
                    {
                        if (j == i) continue;
                        pv[i < j ? pair_pos(i, j, N) : pair_pos(j, i, N)] = 0.0;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < NP; q++) any |= (pv[q] != 0.0);
            if (any)
            {
                for (int it = 1; it <= 25; it++)
                {
                    double pos[N], neg[N];
#pragma unroll
                    for (int i = 0; i < N; i++) { pos[i] = 0.0; neg[i] = 0.0; }
#pragma unroll
                    for (int i = 0; i < N; i++)
#pragma unroll
                        for (int j = i + 1; j < N; j++)
                        {
                            const double w = pv[pair_pos(i, j, N)];
                            if (w < 0.0) { neg[i] += w; pos[j] += -w; }
                            if (w > 0.0) { pos[i] += w; neg[j] += -w; }
                        }
                    bool outside = false;
#pragma unroll
                    for (int i = 0; i < N; i++)
                    {
                        const double vi = (double)val[i];
                        const double newPF = vi + (pos[i] + neg[i]) * dt;
                        double limN = 1.0, limP = 1.0;
                        if (newPF < 0.0) { outside = true; limN = dmin_ref(1.0, -(vi + pos[i] * dt) / (neg[i] * dt)); }
                        if (newPF > 1.0) { outside = true; limP = dmin_ref(1.0, (1.0 - (vi + neg[i] * dt)) / (pos[i] * dt)); }
                        neg[i] = limN;
                        pos[i] = limP;
                    }
                    if (!outside) break;   // every limit is 1
                    bool needed = false;
#pragma unroll
                    for (int i = 0; i < N; i++)
#pragma unroll
                        for (int j = i + 1; j < N; j++)
                        {
                            const int q = pair_pos(i, j, N);
                            if (pv[q] < 0.0)
                            {
                                const double lim = dmin_ref(neg[i], pos[j]);
                                pv[q] *= lim;
                                if (lim < 1.0) needed = true;
                            }
                            if (pv[q] > 0.0)
                            {
                                const double lim = dmin_ref(pos[i], neg[j]);
                                pv[q] *= lim;
                                if (lim < 1.0) needed = true;
                            }
                        }
                    if (!needed) break;
                    if (it == 25) st |= kStLimiterCap;
                }
            }
        }
        // ---- merge (FP64) and finalize --------------------------------------------------------------
        // The reference first zeroes the increments below DBL_EPSILON, then tries them for plausibility
        // (a warning) and then merges those of at least DBL_EPSILON: one pass, since both sums have the
        // same terms in the same order.
        double vd[N];
#pragma unroll
        for (int i = 0; i < N; i++) vd[i] = (double)val[i];
#pragma unroll
        for (int i = 0; i < N; i++)
#pragma unroll
            for (int j = i + 1; j < N; j++)
            {
                const double value = pv[pair_pos(i, j, N)] * dt;
                if (fabs(value) >= DBL_EPSILON)
                {
                    vd[i] += value;
                    vd[j] += -value;
                }
            }
        if (any)
        {
#pragma unroll
            for (int i = 0; i < N; i++)
                if (vd[i] < -(double)FLT_EPSILON || vd[i] > 1.0 + (double)FLT_EPSILON) st |= kStNormalizeWarn;
        }
        const double hi_snap = 1.0 - p.eps_snap;
        const double lo_snap = 0.0 + p.eps_snap;
        double total = 0.0;
        int m = 0;
        bool keep[N];
#pragma unroll
        for (int i = 0; i < N; i++)
        {
            double w = vd[i];
            keep[i] = true;
            if (w >= hi_snap) w = 1.0;
            if (w <= lo_snap) { w = 0.0; keep[i] = false; }
            total += w;
            vd[i] = w;
            m += keep[i];
        }
        const double norm = 1.0 / total;
        int pos = 0;
        if (!mine) continue;
#pragma unroll
        for (int i = 0; i < N; i++)
        {
            if (keep[i])
            {
                const R w = (m > 1) ? (R)(vd[i] * norm) : R(1);
                if (!isfinite((double)w)) st |= kStNonFinite;
                a.idx_out[pos * N_ + v] = (int16_t)g[i];
                vout[pos * N_ + v] = w;
                if (in_volume_window(p, v))
                {
                    const int gi = g[i];
                    const double wi = (double)w;
                    bool hit = false;
#pragma unroll
                    for (int c = 0; c < kVolCache; c++)
                        if (cg[c] == gi) { cv[c] += wi; hit = true; }
                    if (!hit)
                    {
                        if (cg[kVolCache - 1] >= 0)
                            vol_insert_n(s_key, s_sum, kTileVolSlots, a.vol_acc, cg[kVolCache - 1], cv[kVolCache - 1]);
#pragma unroll
                        for (int c = kVolCache - 1; c > 0; c--) { cg[c] = cg[c - 1]; cv[c] = cv[c - 1]; }
                        cg[0] = gi;
                        cv[0] = wi;
                    }
                }
                pos++;
            }
        }
        if (m == 0) st |= kStEmptyVoxel;
        a.cnt_out[v] = (uint8_t)pos;
        eout += pos;
    }
#pragma unroll
    for (int c = 0; c < kVolCache; c++)
        if (cg[c] >= 0) vol_insert_n(s_key, s_sum, kTileVolSlots, a.vol_acc, cg[c], cv[c]);
    flush_block(a, 0u, 0u, eout, st, s_cnt, s_key, s_sum, kTileVolSlots, t, blockDim.x);
}

// ---- anisotropic energies and mobilities -----------------------------------------------------------
// Neighbour of a voxel at offset d without indexing the offset arrays by a runtime value.
__device__ __forceinline__ long long nb_at(const Neighbourhood& nb, const signed char* d)
{
    const long long x = d[0] < 0 ? nb.X[0] : (d[0] > 0 ? nb.X[2] : nb.X[1]);
    const long long y = d[1] < 0 ? nb.Y[0] : (d[1] > 0 ? nb.Y[2] : nb.Y[1]);
    const long long z = d[2] < 0 ? nb.Z[0] : (d[2] > 0 ? nb.Z[2] : nb.Z[1]);
    return x + y + z;
}

// Models of the interface normal need the gradient of every list entry besides the classify kernel's
// list, values and Laplacians.  One thread per wide voxel of list length blockIdx.y + 2: the
// gradients from the neighbours in global memory, in gradient-stencil order as gather_list sums them,
// then list_step with its working arrays (capacity kListCap) in local memory.  Bound: the latency of
// the neighbour loads and of the model functions (pow, acos); in an early solidification one voxel in
// ten is wide, so a warp over the wide voxels instead of over the grid has ten times the lanes at
// work, and the bulk voxels cost the classify kernel's copy only.
template <class R>
__global__ void __launch_bounds__(128) aniso_list_kernel(const __grid_constant__ StepParams p, const StepArrays a,
                                                         int nslices)
{
    __shared__ int s_key[kTileVolSlots];
    __shared__ double s_sum[kTileVolSlots];
    __shared__ unsigned long long s_cnt[3];
    const int n = blockIdx.y + 2, t = threadIdx.x;
    const unsigned* __restrict__ off = a.bucket_off + (long long)n * (nslices + 1);
    const unsigned total = off[nslices];
    const unsigned per = ((total + gridDim.x * blockDim.x - 1u) / (gridDim.x * blockDim.x)) * blockDim.x;
    const unsigned r0 = blockIdx.x * per;
    if (r0 >= total) return;
    const unsigned r1 = min(total, r0 + per);
    for (int i = t; i < kTileVolSlots; i += blockDim.x) { s_key[i] = -1; s_sum[i] = 0.0; }
    if (t < 3) s_cnt[t] = 0ull;
    __syncthreads();
    const long long N = p.n;
    const uint8_t* __restrict__ cnt = a.cnt_in;
    const int16_t* __restrict__ gin = a.idx_in;
    const R* __restrict__ vin = static_cast<const R*>(a.val_in);
    R* __restrict__ vout = static_cast<R*>(a.val_out);
    const int2* __restrict__ buck = a.bucket + (long long)n * a.bucket_cap;
    const int pad = ((2 * n + 7) / 8) * 8;
    uint32_t st = 0;
    unsigned eout = 0;
    for (unsigned e = r0 + t; e < r1; e += blockDim.x)
    {
        const int sl = slice_of(off, nslices, e);
        const int2 ent = buck[(long long)sl * a.slice + (e - off[sl])];
        const unsigned char* __restrict__ wbase = a.wl + (long long)sl * a.wl_slice + ent.y;
        const long long v = ent.x & 0x7fffffff;
        const int flag = (ent.x >> 31) ? 2 : 1;
        const int16_t* __restrict__ rg = reinterpret_cast<const int16_t*>(wbase);
        const R* __restrict__ rv = reinterpret_cast<const R*>(wbase + pad);
        constexpr int KP = kListCap * (kListCap - 1) / 2;
        int16_t g[kListCap];
        R val[kListCap], lap[kListCap], sg[KP], grad[3 * kListCap];
        double pv[KP], pos[kListCap], neg[kListCap];
        for (int k = 0; k < n; k++)
        {
            g[k] = rg[k];
            val[k] = rv[k];
            lap[k] = rv[n + k];
            grad[3 * k] = grad[3 * k + 1] = grad[3 * k + 2] = R(0);
        }
        const Neighbourhood nb(p, v);
        for (int q = 0; q < p.ngs; q++)
        {
            const long long u = nb_at(nb, p.gs_d[q]);
            const int cu = cnt[u];
            for (int s = 0; s < cu; s++)
            {
                const R phi = vin[s * N + u];
                const int gu = gin[s * N + u];
                int f = 0;
                while (f < n && g[f] != gu) f++;
                if (f < n)
                {
                    const R gx = (R)p.gs_w[q][0] * phi;
                    const R gy = (R)p.gs_w[q][1] * phi;
                    const R gz = (R)p.gs_w[q][2] * phi;
                    grad[3 * f] += gx;
                    grad[3 * f + 1] += gy;
                    grad[3 * f + 2] += gz;
                }
            }
        }
        const ListScratch<R> sc{g, val, lap, sg, pv, pos, neg, 1, grad};
        const int m = list_step<R>(p, a, sc, n, flag, st, v, (int)cnt[v]);
        a.cnt_out[v] = (uint8_t)m;
        for (int i = 0; i < m; i++)
        {
            a.idx_out[i * N + v] = g[i];
            vout[i * N + v] = val[i];
            if (in_volume_window(p, v)) vol_insert_n(s_key, s_sum, kTileVolSlots, a.vol_acc, g[i], (double)val[i]);
        }
        eout += m;
    }
    flush_block(a, 0u, 0u, eout, st, s_cnt, s_key, s_sum, kTileVolSlots, t, blockDim.x);
}

// The general-path worklist with anisotropic models: one thread per voxel.
template <class R, int KS, int KL>
__global__ void __launch_bounds__(64) aniso_worklist_kernel(const __grid_constant__ StepParams p, const StepArrays a)
{
    __shared__ int s_key[kTileVolSlots];
    __shared__ double s_sum[kTileVolSlots];
    __shared__ unsigned long long s_cnt[3];
    for (int i = threadIdx.x; i < kTileVolSlots; i += blockDim.x) { s_key[i] = -1; s_sum[i] = 0.0; }
    if (threadIdx.x < 3) s_cnt[threadIdx.x] = 0ull;
    __syncthreads();
    const unsigned total = min(*a.slow_count, a.slow_cap);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.counters[kCntGeneralLast], (unsigned long long)total);
    uint32_t st = 0;
    unsigned eo = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
    {
        unsigned wide = 0, ein = 0, eout = 0;   // wide and ein were counted by the classify kernel
        voxel_step_generic<R, KS, KL, true>(p, a, a.slow_list[i], s_key, s_sum, kTileVolSlots, wide, ein, eout, st, false);
        eo += eout;
    }
    flush_block(a, 0u, 0u, eo, st, s_cnt, s_key, s_sum, kTileVolSlots, threadIdx.x, blockDim.x);
}

// Fork of the side streams from a context's stream, and their join into it.  join() is called on
// every path that launched on them, so that no work of a step outlives the step's place in the
// context's stream.
struct SideFork {
    const SideStreams* side;
    cudaStream_t main;
    cudaError_t err = cudaSuccess;

    SideFork(const SideStreams* side_, cudaStream_t s) : side(side_), main(s)
    {
        if (!side) return;
        err = cudaEventRecord(static_cast<cudaEvent_t>(side->fork), main);
        for (int k = 0; k < kSideStreams && err == cudaSuccess; k++)
            err = cudaStreamWaitEvent(on(k), static_cast<cudaEvent_t>(side->fork), 0);
        if (err != cudaSuccess) side = nullptr;   // nothing forked is used
    }
    cudaStream_t on(int k) const { return side ? static_cast<cudaStream_t>(side->stream[k]) : main; }
    cudaError_t join() const
    {
        if (!side) return err;
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < kSideStreams; k++)
        {
            cudaError_t q = cudaEventRecord(static_cast<cudaEvent_t>(side->join[k]), on(k));
            if (q == cudaSuccess) q = cudaStreamWaitEvent(main, static_cast<cudaEvent_t>(side->join[k]), 0);
            if (e == cudaSuccess) e = q;
        }
        return e;
    }
};

// The per-length kernels, dealt out to streams of about equal length (64^3: the longest alone).
template <class R, bool AVG>
void launch_lists(const StepParams& p, const StepArrays& a, int cb, int nblocks, const SideFork& fork, bool together)
{
    const cudaStream_t s = fork.main;
    list_compute_kernel<R, 8, AVG><<<cb, 128, 0, fork.on(0)>>>(p, a, nblocks, together);
    list_compute_kernel<R, 7, AVG><<<cb, 128, 0, fork.on(1)>>>(p, a, nblocks, together);
    list_compute_kernel<R, 6, AVG><<<cb, 128, 0, s>>>(p, a, nblocks, together);
    list_compute_kernel<R, 5, AVG><<<cb, 128, 0, fork.on(3)>>>(p, a, nblocks, together);
    list_compute_kernel<R, 4, AVG><<<cb, 128, 0, s>>>(p, a, nblocks, together);
    list_compute_kernel<R, 3, AVG><<<cb, 128, 0, fork.on(3)>>>(p, a, nblocks, together);
    list_compute_kernel<R, 2, AVG><<<cb, 128, 0, fork.on(1)>>>(p, a, nblocks, together);
}

template <class R, int KS, int KL, int NS>
int launch_tiled_ns(const StepParams& p, const StepArrays& a, void* stream, LaunchInfo* info)
{
    using Smem = TileSmem<R, kTileTY>;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int xchunk = 0, gz = 0, gy = 0, gx = 0;
    tiled_geometry(p.nx, p.ny, p.nz, (int)sizeof(R), &xchunk, &gz, &gy, &gx);
    const int nblocks = gz * gy * gx;
    constexpr bool kSingle = sizeof(R) == 4;
    auto kern = kSingle && !p.aniso && !a.avg_mask ? tile_classify_kernel<R, kTileTY, NS, kSingle>
                                                  : tile_classify_kernel<R, kTileTY, NS, false>;
    const size_t smem = sizeof(Smem);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    auto gk = warp_general_kernel<R, KS, KL>;
    const size_t wsm = 4 * sizeof(WarpScratch<R, KL>);
    e = cudaFuncSetAttribute(gk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wsm);
    if (e != cudaSuccess) return (int)e;
    e = cudaMemsetAsync(a.slow_count, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return (int)e;
    kern<<<dim3(gz, gy, gx), dim3(kTileZ, kTileTY), smem, s>>>(p, a, xchunk);
    if (info && info->after_classify)
    {
        e = cudaEventRecord(static_cast<cudaEvent_t>(info->after_classify), s);
        if (e != cudaSuccess) return (int)e;
    }
    bucket_scan_kernel<<<kListCap - 1, 1024, 0, s>>>(a, nblocks);
    const int cb = compute_blocks(p.n);
    const bool lists_beside = info && info->side && info->worklist < kListsBeside;
    const bool general_beside = lists_beside && info->worklist < kGeneralBeside;
    if (!p.aniso && !general_beside) gk<<<148 * 4, 128, wsm, s>>>(p, a);
    const SideFork fork(lists_beside ? info->side : nullptr, s);
    if (p.aniso)
    {
        aniso_worklist_kernel<R, KS, KL><<<148 * 8, 64, 0, fork.on(0)>>>(p, a);
        aniso_list_kernel<R><<<dim3(cb, kListCap - 1), 128, 0, s>>>(p, a, nblocks);
    }
    else
    {
        if (general_beside) gk<<<148 * 4, 128, wsm, fork.on(2)>>>(p, a);
        const bool together = info && info->worklist > (unsigned long long)p.n / kTogetherShare;
        if (a.avg_mask) launch_lists<R, true>(p, a, cb, nblocks, fork, together);
        else launch_lists<R, false>(p, a, cb, nblocks, fork, together);
    }
    if ((e = fork.join()) != cudaSuccess) return (int)e;
    if (info) info->kernels += p.aniso ? 4 : 10;
    return (int)cudaGetLastError();
}

// The classify kernel and the bucket scan (work records, length buckets and their offsets,
// general-path worklist, bulk copies): the adjoint reverses the lists they leave.  Returns the number of classify blocks (the slices of
// the buckets) or a negative error.
template <class R, int NS>
int launch_classify_ns(const StepParams& p, const StepArrays& a, void* stream)
{
    using Smem = TileSmem<R, kTileTY>;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int xchunk = 0, gz = 0, gy = 0, gx = 0;
    tiled_geometry(p.nx, p.ny, p.nz, (int)sizeof(R), &xchunk, &gz, &gy, &gx);
    auto kern = tile_classify_kernel<R, kTileTY, NS, sizeof(R) == 4>;
    const size_t smem = sizeof(Smem);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return -(int)e;
    e = cudaMemsetAsync(a.slow_count, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return -(int)e;
    kern<<<dim3(gz, gy, gx), dim3(kTileZ, kTileTY), smem, s>>>(p, a, xchunk);
    bucket_scan_kernel<<<kListCap - 1, 1024, 0, s>>>(a, gz * gy * gx);
    e = cudaGetLastError();
    return e == cudaSuccess ? gz * gy * gx : -(int)e;
}

template <class R>
int launch_classify(const StepParams& p, const StepArrays& a, void* stream)
{
    return p.ns == 27 ? launch_classify_ns<R, 27>(p, a, stream) : launch_classify_ns<R, 7>(p, a, stream);
}

template <class R, int KS, int KL>
int launch_tiled(const StepParams& p, const StepArrays& a, void* stream, LaunchInfo* info)
{
    if (p.ns == 27) return launch_tiled_ns<R, KS, KL, 27>(p, a, stream, info);
    if (p.ns == 7) return launch_tiled_ns<R, KS, KL, 7>(p, a, stream, info);
    return -1;
}

template <class R>
int launch_step(const StepParams& p, const StepArrays& a, int k_slots, int variant, void* stream,
                LaunchInfo* info)
{
    if (variant == kVariantGeneric)
    {
        if (info) info->kernels += 1;
        return launch_step_generic<R>(p, a, k_slots, stream);
    }
    switch (k_slots)
    {
        case 8:  return launch_tiled<R, 8, 16>(p, a, stream, info);
        case 12: return launch_tiled<R, 12, 20>(p, a, stream, info);
        case 16: return launch_tiled<R, 16, 24>(p, a, stream, info);
        default: return -1;
    }
}

}  // namespace opgpu
