// Device-side data layout and launch interface of the fused multiphase-field step.
//
// State (one buffer of a ping-pong pair), structure of arrays over N = nx*ny*nz voxels:
//   cnt[N]        uint8   number of stored (positive) fields of the voxel
//   idx[K][N]     int16   grain index of slot s        (slot plane s at idx + s*N)
//   val[K][N]     real    phase-field value of slot s  (real = double or float)
// Slots s >= cnt[v] are never read.  Only positive entries are stored (what NodePF holds after
// NodePF::finalize); the zero-valued candidate entries the reference appends in
// CalculateDerivativesSR are re-derived inside the step kernel from the 3x3x3 neighbourhood.
// A voxel's interface flag is never stored: flag = 2 if cnt > 1, else 1 if any of its 26 periodic
// neighbours has cnt > 1, else 0 (identical to NodePF::finalize + PhaseField::SetFlagsSR).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <vector_types.h>

namespace opgpu {

constexpr int kMaxPhases = 8;

enum : uint32_t {
    kStOverflowK = 1u << 0,
    kStOverflowList = 1u << 1,
    kStEmptyVoxel = 1u << 2,
    kStNormalizeWarn = 1u << 3,
    kStLimiterCap = 1u << 4,
    kStNonFinite = 1u << 5,
    kStAdjointMismatch = 1u << 6,   // the recomputed step does not reproduce the stored next state
};

// Driving-force averaging (average.cu): one bit per pair of stored fields of every interface voxel,
// whether the pair's weight is above the threshold somewhere in the sphere.  Pair (a, b), a < b, of
// the stored fields has bit b(b-1)/2 + a, whatever the voxel's count; word w of voxel v at
// mask[w*N + v] (only the words that a voxel's pairs need are written).
constexpr int kAvgWords = 4;     // 120 pairs of 16 stored fields
struct AvgArrays {
    unsigned* strong;            // [N] key of the voxel's pair above the threshold
    unsigned* mask;              // [kAvgWords][N]
    unsigned* tiles;             // [2 + average_tiles] the tiles searched directly: their number, the next item
                                 // of work, the tiles
    const char4* offsets;        // [noff] sphere offsets with Range - |d| > 0, nearest first
    int noff;
    int range;
    double weight_threshold;     // sqrt(Threshold (1 - Threshold))
};

// counters[] slots: the step kernel adds into the per-step slots 0-2; the grain-update kernel rolls
// them into the running totals and clears them.
enum {
    kCntWide = 0, kCntEntriesIn = 1, kCntEntriesOut = 2, kCntOverflowVoxels = 3,
    kCntWideTotal = 4, kCntEntriesInTotal = 5, kCntEntriesOutTotal = 6, kCntWideLast = 7, kCntSteps = 8,
    kCntGeneralLast = 9,      // voxels the last step sent through the general per-voxel path
    kCntGeneralTotal = 10,
    kCntCrowdedLast = 11,     // of those, voxels whose window held more grains than slots
    kCntCrowdedTotal = 12,
    kNumCounters = 13
};

// Bytes of a work-list record with n fields of type R: grains padded to 8 bytes, values, Laplacians.
__host__ __device__ constexpr int work_record_bytes(int n, int rsz) { return ((2 * n + 7) / 8) * 8 + 2 * n * rsz; }

struct StepParams {
    int nx, ny, nz;
    long long n;
    // Laplacian stencil (LaplacianStencil::Set order) and the neighbour set used to discover
    // candidates after it (GradientStencil::Set order), both with periodic offsets.
    int ns;
    signed char lap_d[27][3];
    double lap_w[27];
    int ng;
    signed char grad_d[27][3];
    double pref_do;          // Pi^2/Eta^2 (DoubleObstacle.cpp:504)
    double pref_df;          // Pi/Eta     (DrivingForce.cpp:507)
    double dt;
    double eps_snap;         // finalize snap/erase threshold (DBL_EPSILON in the FP64 form)
    int nphases;
    double sigma_p[kMaxPhases * kMaxPhases];
    double mu_p[kMaxPhases * kMaxPhases];
    double allowed_p[kMaxPhases * kMaxPhases];   // Limit*Prefactor*MaxEnergy*RegularizationFactor
    int limiting;
    double tj_factor;
    int consider_nucleus_volume;
    int pair_mode;           // OPGPU_PAIRS_*
    unsigned long long hash_seed;
    double hash_lo, hash_span;
    int ngrains;
    int use_dg;
    // anisotropic interface energy (InterfaceProperties::SetSR, src/InterfaceProperties.cpp:617-673):
    // per phase pair the model (0 ISO, 1 CUBIC, 2 DISORIENTATION, 3 HEXBOETTGER, 4 HEXSUN, 5 HEXYANG),
    // its Epsilon1 (eps_p) and Epsilon2..4 (eps_x) and MaxEnergy; per phase solid (1) or
    // liquid (0); the gradient stencil in GradientStencil::Set order with its weights per axis
    int aniso;
    signed char emodel[kMaxPhases * kMaxPhases];
    double eps_p[kMaxPhases * kMaxPhases];
    double eps_x[kMaxPhases * kMaxPhases][3];
    int facet_lo[kMaxPhases * kMaxPhases], facet_hi[kMaxPhases * kMaxPhases];   // FACETED: rows of facets
    signed char mmodel[kMaxPhases * kMaxPhases];   // mobility model per phase pair (codes of emodel)
    int mfacet_lo[kMaxPhases * kMaxPhases], mfacet_hi[kMaxPhases * kMaxPhases];   // FACETED mobility rows
    double meps[kMaxPhases * kMaxPhases][4];       // its Epsilon1..4
    double maxe_p[kMaxPhases * kMaxPhases];
    signed char solid_p[kMaxPhases];
    int ngs;
    signed char gs_d[27][3];
    double gs_w[27][3];
    // x-planes [vol_x0, vol_x1) count in the grain volumes (all planes unless a slab of a larger
    // grid: its halo planes are excluded)
    int vol_x0, vol_x1;
};

// Whether voxel v lies in the planes that count in the grain volumes.
__device__ __forceinline__ bool in_volume_window(const StepParams& p, long long v)
{
    if (p.vol_x0 == 0 && p.vol_x1 == p.nx) return true;
    const int x = (int)(v / ((long long)p.ny * p.nz));
    return x >= p.vol_x0 && x < p.vol_x1;
}

struct StepArrays {
    const uint8_t* cnt_in;
    const int16_t* idx_in;
    const void* val_in;
    uint8_t* cnt_out;
    int16_t* idx_out;
    void* val_out;
    const double* vr;          // [G] VolumeRatio
    const int16_t* gphase;     // [G]
    const int8_t* gstage;      // [G]
    const double* dg;          // [G] or null
    const double* pair_sigma;  // [G*G] or null
    const double* pair_mu;     // [G*G] or null
    const double* dg_pair;     // [G*G] limited driving force per grain pair, or null (evaluated in place)
    const unsigned* avg_mask;  // [kAvgWords][N] AvgArrays::mask, or null without averaging
    const double* grot;        // [G*9] grain rotation matrices (row-major), for anisotropic energies
    double* vol_acc;           // [G] volume accumulator of the output state (zeroed by the caller)
    uint32_t* status;          // soft status bits
    unsigned long long* counters;  // kNumCounters
    // overflow worklist of the tiled kernel (voxels whose lists exceed its register capacity)
    int* slow_list;            // [slow_cap]
    unsigned* slow_count;      // reset by the launcher before every step
    unsigned slow_cap;
    // work buffer between the classify kernel and the per-length compute kernels: every list is a
    // record of n fields (int16 grains padded to 8 bytes, then n values, then n Laplacians) packed
    // in its classify block's byte slice; bucket entries (voxel | flag2 << 31, record offset)
    unsigned char* wl;         // [blocks][wl_slice] bytes
    long long wl_slice;        // bytes per classify block
    int2* bucket;              // [kListCap + 1][bucket_cap] entries per list length, block-private slices
    unsigned* bucket_count;    // [kListCap + 1][max blocks] entries per slice
    unsigned* bucket_off;      // [kListCap + 1][blocks + 1] exclusive prefix of bucket_count per list
                               // length, then the length's total
    const double* facets;      // FACETED: rows of (unit facet normal x, y, z, SigmaF, EpsilonEF)
    long long bucket_cap;
    int slice;                 // entries per classify-block slice
};

constexpr int kListCap = 8;    // list capacity of the split kernels (longer lists: overflow worklist)
constexpr int kTileCols = 16;  // tile of the classify kernel: kTileCols (z) x kTileRows (y) voxels,
constexpr int kTileRows = 8;   // one thread each

// Launch geometry of the classify kernel: tiles of kTileCols (z) x kTileRows (y) voxels marching over
// `xchunk` x-planes.  A block loads xchunk + 2 planes and spends about one more on setting up its
// shared memory; the device holds 148 SMs x 3 (FP64) or 5 (FP32) blocks at a time.  The estimate is
// planes times waves, plus a third of a wave for blocks over bulk and over interfaces that differ in
// length; the shortest wins.  Measured, classify in us (chunk): FP64 64^3 81 (2) 62 (5); 96^3 181 (5) 151
// (8) 140 (16); 128^3 318 (13) 345 (16) 372 (43); 160^3 566 (15) 577 (20); FP32 150x97x203, 7-point 376
// (15) 365 (21) 341 (38).  The estimate's choice is the fastest measured one each time (13 at 128^3, where
// it ranks 43 before 16, the other way round than measured).  slice = voxels one block can append to a
// bucket.
inline void tiled_geometry(int nx, int ny, int nz, int real_size, int* xchunk, int* gz, int* gy, int* gx)
{
    const int tzb = (nz + kTileCols - 1) / kTileCols, tyb = (ny + kTileRows - 1) / kTileRows;
    const long long tiles = (long long)tzb * tyb, resident = 148 * (real_size == 8 ? 3 : 5);
    long long best = 0;
    int xc = 2;
    for (int c = 2; c <= 64 && c <= nx + 1; c++)
    {
        const long long blocks = tiles * ((nx + c - 1) / c);
        const long long waves = (blocks + resident - 1) / resident;
        const long long cost = (c + 3) * (20 * waves + 7);
        if (best == 0 || cost < best) { best = cost; xc = c; }
    }
    *xchunk = xc;
    *gz = tzb;
    *gy = tyb;
    *gx = (nx + xc - 1) / xc;
}

enum { kVariantTiled = 0, kVariantGeneric = 1 };

// Side streams of a context: independent kernels of one step run beside each other between a fork
// from and a join into the context's stream.
constexpr int kSideStreams = 4;
struct SideStreams {
    void* stream[kSideStreams] = {};   // cudaStream_t
    void* fork = nullptr;              // cudaEvent_t
    void* join[kSideStreams] = {};     // cudaEvent_t
};

// Which kernels of a step run beside each other goes by the length of the general-path worklist, as the
// host last read it (with the status word).  All write disjoint voxels; the order changes no result.
// Each per-length kernel is a chain of dependent arithmetic and instruction fetches whose length hardly
// depends on its entry count on small grids (64^3, FP64: 17, 19, 26, 34, 54, 77, 115 us for N = 2..8), so
// that they gain from each other's company until each fills the device.  The general path has the
// opposite: it gathers from the whole neighbourhood, and once it runs long the lists beside it cost it
// its cache.  Step in us, one after another / lists beside each other / general path beside them (mean
// grain volume, worklist):
//   FP64  64^3 8389       <1 k   289   183   149      FP32  64^3 8389       <1 k   290   178   143
//         128^3 8389       4 k   842   638   621            128^3 8389       4 k   801   593   582
//         192^3 8389      14 k  1921  1765  1832            192^3 8389      14 k  1753  1623  1632
//         256^3 8389      29 k  4073  4028  4133            256^3 8389      29 k  3771  3708  3748
//         128^3 3500      31 k  1485  1344  1466            128^3 3500      31 k  1371  1234  1261
//         64^3 1728       47 k   985   931   950            160^3 3500      61 k  2227  2093  2300
//         240^3 5000      83 k  5016  5008  5623            240^3 5000      83 k  4680  4831  4832
//         224^3 3500     180 k  7065  7419  8199            224^3 3500     180 k  6313  6758  7310
//         96^3 1728      170 k  2927  3008  3383            96^3 1728      100 k  2118  2255  2296
// The adjoint's lists (one after another / worklist kernel beside them / all beside each other, us):
//   FP64 96^3 8192 2 k 2573 2259 2167; 96^3 4000 9 k 5127 5009 5267; 128^3 8192 4 k 2969 2641 2779;
//   192^3 8192 14 k 7365 7105 7464; 224^3 4000 120 k 20409 20588 21262; 256^3 4000 180 k 34234 36768 39128.
// The tangent step gains with all of them beside each other at every size (96^3 1924 -> 1145, 256^3 17141 ->
// 16183).
constexpr unsigned kGeneralBeside = 10000;      // below: the general path beside the lists
constexpr unsigned kListsBeside = 80000;        // below: the lists beside each other
constexpr unsigned kAdjointListsBeside = 2500;  // below: the adjoint's lists beside each other
// Before a first step: the worklist of grains of some 8400 voxels.
inline unsigned worklist_guess(long long n) { return (unsigned)(n / 500); }

// Filled by the launchers: kernels launched, and an event recorded after the classify kernel
// (when `after_classify` is not null) so the caller can time it separately.
struct LaunchInfo {
    void* after_classify = nullptr;   // cudaEvent_t
    const SideStreams* side = nullptr;   // null: every kernel on the context's stream
    unsigned worklist = 0;            // length of the general-path worklist, as last known
    int kernels = 0;
};

// Launchers (defined in step_f64.cu / step_f32.cu).  k_slots in {8, 12, 16}; variant selects the
// tiled production kernel or the full-grid generic kernel (same results, used for validation).
int launch_step_f64(const StepParams& p, const StepArrays& a, int k_slots, int variant, void* stream,
                    LaunchInfo* info);
int launch_step_f32(const StepParams& p, const StepArrays& a, int k_slots, int variant, void* stream,
                    LaunchInfo* info);
// The classify kernel of the tiled step alone; returns the number of classify blocks or < 0.
int launch_classify_f64(const StepParams& p, const StepArrays& a, void* stream);
int launch_classify_f32(const StepParams& p, const StepArrays& a, void* stream);
// Driving-force averaging of a state (average.cu): writes aa.strong, aa.mask and aa.tiles; adds its launches
// to *kernels.
size_t average_tiles(int nx, int ny, int nz);
int launch_average(const StepParams& p, const AvgArrays& aa, const uint8_t* cnt, const int16_t* idx,
                   const void* val, bool fp32, const double* vr, void* stream, int* kernels);
// Add the volumes of the window planes of a state to vol_acc (defined in step_f64.cu).
int launch_volume_recount(const StepParams& p, const uint8_t* cnt, const int16_t* idx, const void* val, int fp32,
                          double* vol_acc, void* stream);

}  // namespace opgpu
