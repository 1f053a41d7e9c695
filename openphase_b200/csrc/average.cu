// Driving-force averaging: DrivingForce::Average with $Average Yes (src/DrivingForce.cpp:242-256),
// the reference default.  For the per-grain driving force, every interface voxel's pair (A, B)
// carries raw = dG_B - dG_A (A before B in the voxel's list) and weight sqrt(phi_A phi_B)
// (SetWeights, :276-291; PHASEFIELDS weights, the default, :59, :137).  The reference makes two
// passes over a sphere of radius Range around each interface voxel:
//   collect    (CollectAverage, :293-383): for a pair whose weight exceeds Threshold' * VR_A VR_B
//              (Threshold' = sqrt(t (1 - t))), tmp = sum(w_u raw_u) / sum(w_u) over the sphere's
//              voxels holding the pair;
//   distribute (DistributeAverage, :384-478): for every pair of positive fields, average =
//              sum(w_u tmp_u) / sum(w_u) over the sphere's voxels where the pair's weight exceeds
//              the threshold, else the voxel's own tmp (0 when the pair is below it there).
// raw depends on the grain pair alone, not on the voxel, and both passes use one threshold, so both
// averages are averages of equal values: the result is raw itself when some voxel of the sphere has
// the pair above the threshold, and 0 when none has.  What is left to compute is that decision,
// one bit per stored pair and voxel; the step then takes the pair's limited force from its per-pair
// table (the C library's tanh, as the reference's limiter :548-583) or none (pair_force).  The sums
// the reference forms differ from raw by their rounding only (some 1e-16 of it).
//
// Kernels: df_mark_kernel writes per voxel the key of its pair above the threshold (at most one
// unless the threshold is low: then "several", resolved from the lists).  df_reach_kernel owns a
// tile of voxels: it collects the marks of the tile and its halo once, sorted by key, so that a
// pair of a voxel is tested against the marked voxels of its own key only (some tens) instead of
// against the whole sphere (925 offsets at radius 6).  A tile whose halo holds a "several" or more marks
// or keys than the tables take is left at once and listed; df_tiles_kernel searches the sphere directly
// for the voxels of the listed tiles, nearest offsets first (search_sphere), spread over the whole
// device.  Radii above kReachRange go to the direct search at once.
//
// Measured (B200, 96^3, 105 grains, radius 6, FP64, per step): the two passes over the sphere
// 4232 + 40214 us; the direct search of every voxel about 2900 us; sorted marks 474 us, df_mark 30 us,
// and the step itself runs on the tiled kernels (45.6 -> 0.90 ms in all).  Where tables overflow (steps in
// ms, searched by the tile's own block -> by df_tiles_kernel): radius 16 with 105 grains 84.7 -> 38.5, with
// 30 grains 52.7 -> 21.1; 400 grains (VolumeRatio < 1: "several" in every halo), radius 6, 17.6 -> 10.4.
#include <cfloat>
#include <cstdint>

#include "opgpu_device.h"
#include "step_kernel.cuh"

namespace opgpu {

namespace {

constexpr unsigned kSeveral = 0xFFFFFFFFu;

// Key of an unordered grain pair (grain indices are below 2^15), never 0 or kSeveral.
__device__ __forceinline__ unsigned pair_code(int A, int B)
{
    const unsigned lo = A < B ? A : B, hi = A < B ? B : A;
    return (lo << 15 | hi) + 1u;
}

// Whether interface voxel u (c stored fields) has the pair (A, B) above the threshold.
template <class R>
__device__ bool above(const uint8_t* __restrict__ cnt, const int16_t* __restrict__ idx, const R* __restrict__ val,
                      long long N, long long u, int A, int B, double thr)
{
    const int c = cnt[u];
    int sa = -1, sb = -1;
    for (int k = 0; k < c; k++)
    {
        const int g = idx[k * N + u];
        if (g == A) sa = k;
        if (g == B) sb = k;
    }
    return sa >= 0 && sb >= 0 && sqrt((double)val[sa * N + u] * (double)val[sb * N + u]) > thr;
}

template <class R>
__global__ void __launch_bounds__(256) df_mark_kernel(long long N, double threshold, const uint8_t* __restrict__ cnt,
                                                       const int16_t* __restrict__ idx, const R* __restrict__ val,
                                                       const double* __restrict__ vr, unsigned* __restrict__ strong,
                                                       unsigned* __restrict__ tiles)
{
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= N) return;
    if (v < 2) tiles[v] = 0u;   // no tile listed, none searched
    const int c = cnt[v];
    unsigned key = 0;
    for (int b = 1; b < c; b++)
    {
        const int B = idx[b * N + v];
        const double wb = (double)val[b * N + v];
        for (int a = 0; a < b; a++)
        {
            const int A = idx[a * N + v];
            if (sqrt((double)val[a * N + v] * wb) > threshold * (vr[A] * vr[B])) key = key ? kSeveral : pair_code(A, B);
        }
    }
    strong[v] = key;
}

// The voxel at offset d of (x, y, z); |d| per axis is below the grid's extent.
__device__ __forceinline__ long long sphere_voxel(const StepParams& p, unsigned plane, int x, int y, int z, char4 d)
{
    int ux = x + d.x, uy = y + d.y, uz = z + d.z;
    ux = ux < 0 ? ux + p.nx : (ux >= p.nx ? ux - p.nx : ux);
    uy = uy < 0 ? uy + p.ny : (uy >= p.ny ? uy - p.ny : uy);
    uz = uz < 0 ? uz + p.nz : (uz >= p.nz ? uz - p.nz : uz);
    return (long long)ux * plane + uy * p.nz + uz;
}

constexpr int kFewFields = 4, kFewPairs = kFewFields * (kFewFields - 1) / 2;

// The mask of voxel v = (x, y, z) by the direct search.
template <class R>
__device__ __noinline__ void search_sphere(const StepParams& p, const AvgArrays& aa, const uint8_t* __restrict__ cnt,
                                           const int16_t* __restrict__ idx, const R* __restrict__ val,
                                           const double* __restrict__ vr, int x, int y, int z)
{
    const long long N = p.n;
    const unsigned plane = (unsigned)p.ny * (unsigned)p.nz;
    const long long v = (long long)x * plane + y * p.nz + z;
    const int c = cnt[v];
    if (c < 2) return;
    const int np = c * (c - 1) / 2;
    if (c <= kFewFields)
    {
        // the usual case: all pair codes in registers, the keys of four offsets in flight
        unsigned code[kFewPairs];
        int g[kFewFields];
#pragma unroll
        for (int k = 0; k < kFewFields; k++) g[k] = k < c ? idx[k * N + v] : 0;
#pragma unroll
        for (int b = 1; b < kFewFields; b++)
#pragma unroll
            for (int a = 0; a < b; a++) code[b * (b - 1) / 2 + a] = b < c ? pair_code(g[a], g[b]) : 0u;
        const unsigned full = (1u << np) - 1u;
        unsigned found = 0;
        for (int q0 = 0; q0 < aa.noff && found != full; q0 += 4)
        {
            unsigned key[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                key[k] = q0 + k < aa.noff ? aa.strong[sphere_voxel(p, plane, x, y, z, aa.offsets[q0 + k])] : 0u;
#pragma unroll
            for (int k = 0; k < 4; k++)
            {
                if (key[k] == 0u) continue;
                if (key[k] != kSeveral)
                {
#pragma unroll
                    for (int i = 0; i < kFewPairs; i++) found |= key[k] == code[i] ? 1u << i : 0u;
                    continue;
                }
                const long long u = sphere_voxel(p, plane, x, y, z, aa.offsets[q0 + k]);
                for (int b = 1, bit = 0; b < c; b++)
                    for (int a = 0; a < b; a++, bit++)
                    {
                        const int A = idx[a * N + v], B = idx[b * N + v];
                        if (!((found >> bit) & 1u) && above<R>(cnt, idx, val, N, u, A, B, aa.weight_threshold * (vr[A] * vr[B])))
                            found |= 1u << bit;
                    }
            }
        }
        aa.mask[v] = found;
        return;
    }
    for (int w = 0; w * 32 < np; w++)
    {
        // the pairs of this word of the mask: positions 32w .. 32w + 31 in the order (0,1) (0,2)
        // (1,2) (0,3) .., all searched in one walk over the sphere
        const int m = min(32, np - 32 * w);
        const unsigned full = m == 32 ? 0xFFFFFFFFu : (1u << m) - 1u;
        unsigned found = 0;
        for (int q = 0; q < aa.noff; q++)
        {
            const long long u = sphere_voxel(p, plane, x, y, z, aa.offsets[q]);
            const unsigned key = aa.strong[u];
            if (key == 0u) continue;
            int b = 1, at = -32 * w;   // position of (0, b) relative to this word
            for (; at + b <= 0; b++) at += b;
            for (; b < c && at < m; at += b, b++)
            {
                const int B = idx[b * N + v];
                // a key holds B or it matches no pair (a, b)
                const unsigned lo = (key - 1u) >> 15, hi = (key - 1u) & 0x7FFFu;
                if (key != kSeveral && lo != (unsigned)B && hi != (unsigned)B) continue;
                for (int a = 0; a < b; a++)
                {
                    const int bit = at + a;
                    if (bit < 0 || bit >= m || ((found >> bit) & 1u)) continue;
                    const int A = idx[a * N + v];
                    const bool hit = key == kSeveral
                                         ? above<R>(cnt, idx, val, N, u, A, B, aa.weight_threshold * (vr[A] * vr[B]))
                                         : key == pair_code(A, B);
                    if (hit) found |= 1u << bit;
                }
            }
            if (found == full) break;
        }
        aa.mask[(long long)w * N + v] = found;
    }
}

template <class R>
__global__ void __launch_bounds__(128) df_sphere_kernel(const __grid_constant__ StepParams p, AvgArrays aa,
                                                         const uint8_t* __restrict__ cnt,
                                                         const int16_t* __restrict__ idx, const R* __restrict__ val,
                                                         const double* __restrict__ vr)
{
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= p.n) return;
    const int z = (int)(v % p.nz), y = (int)((v / p.nz) % p.ny), x = (int)(v / ((long long)p.ny * p.nz));
    search_sphere<R>(p, aa, cnt, idx, val, vr, x, y, z);
}

// Tile of df_reach_kernel (x, y, z) and its tables.  Halo positions are packed 10 bits an axis.
constexpr int kReachX = 8, kReachY = 8, kReachZ = 16;
// Largest radius the tiles are tried for.  Whether the tables hold a halo depends on how many marks it has:
// while they do a step takes a third to a tenth of the direct search's time (96^3, radius 12: 0.9 ms against
// 5.8 with 8 grains, 0.8 against 8.2 with 30), and where they do not it takes 0.8 to 1.13 times that time
// (radius 13 to 16, 8 to 400 grains).  Above 16 no measured halo fits.
constexpr int kReachRange = 16;
constexpr int kReachMarks = 4608;   // at radius 6 a halo has 11200 voxels, some 20 % of them marked
constexpr int kReachKeys = 256;

__device__ __forceinline__ int wrap_axis(int i, int n)
{
    i %= n;
    return i < 0 ? i + n : i;
}

template <class R>
__global__ void __launch_bounds__(256) df_reach_kernel(const __grid_constant__ StepParams p, AvgArrays aa,
                                                        const uint8_t* __restrict__ cnt,
                                                        const int16_t* __restrict__ idx, const R* __restrict__ val,
                                                        const double* __restrict__ vr)
{
    __shared__ unsigned key_of[kReachKeys];       // hash of the halo's keys (0: free)
    __shared__ int first[kReachKeys + 1];         // marks of each key: their count, then their first place
    __shared__ int filled[kReachKeys];
    __shared__ unsigned entry[kReachMarks];       // marked halo positions
    __shared__ uint8_t slot_of[kReachMarks];      // and the hash slots of their keys
    __shared__ unsigned place[kReachMarks];       // halo positions sorted by key
    __shared__ int entries, failed;
    const int t = threadIdx.x, NT = blockDim.x, r = aa.range;
    const int x0 = blockIdx.z * kReachX, y0 = blockIdx.y * kReachY, z0 = blockIdx.x * kReachZ;
    const int hx = kReachX + 2 * r, hy = kReachY + 2 * r, hz = kReachZ + 2 * r;
    const long long N = p.n;
    const unsigned plane = (unsigned)p.ny * (unsigned)p.nz;
    for (int i = t; i < kReachKeys; i += NT) { key_of[i] = 0u; first[i] = 0; filled[i] = 0; }
    if (t == 0) { entries = 0; failed = 0; }
    __syncthreads();
    for (int i = t; i < hx * hy * hz && !*(volatile int*)&failed; i += NT)
    {
        const int iz = i % hz, iy = (i / hz) % hy, ix = i / (hz * hy);
        const long long u = (long long)wrap_axis(x0 - r + ix, p.nx) * plane + wrap_axis(y0 - r + iy, p.ny) * p.nz
                          + wrap_axis(z0 - r + iz, p.nz);
        const unsigned key = aa.strong[u];
        if (key == 0u) continue;
        const int e = atomicAdd(&entries, 1);
        if (key == kSeveral || e >= kReachMarks) { failed = 1; continue; }
        unsigned h = (key * 2654435761u) >> 24;
        int probe = 0;
        for (; probe < kReachKeys; probe++)
        {
            const unsigned k = atomicCAS(&key_of[h], 0u, key);
            if (k == 0u || k == key) break;
            h = (h + 1) & (kReachKeys - 1);
        }
        if (probe == kReachKeys) { failed = 1; continue; }
        atomicAdd(&first[h], 1);
        entry[e] = (unsigned)(ix << 20 | iy << 10 | iz);
        slot_of[e] = (uint8_t)h;
    }
    __syncthreads();
    if (failed)
    {
        if (t == 0) aa.tiles[2u + atomicAdd(&aa.tiles[0], 1u)] = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        return;
    }
    if (t < 32)
    {
        // exclusive scan of the counts by one warp
        int carry = 0;
        for (int b = 0; b < kReachKeys; b += 32)
        {
            const int n = first[b + t];
            int incl = n;
            for (int o = 1; o < 32; o <<= 1)
            {
                const int q = __shfl_up_sync(0xffffffffu, incl, o);
                if (t >= o) incl += q;
            }
            first[b + t] = carry + incl - n;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (t == 0) first[kReachKeys] = carry;
    }
    __syncthreads();
    const int total = entries;
    for (int e = t; e < total; e += NT)
    {
        const int h = slot_of[e];
        place[first[h] + atomicAdd(&filled[h], 1)] = entry[e];
    }
    __syncthreads();
    for (int i = t; i < kReachX * kReachY * kReachZ; i += NT)
    {
        const int iz = i % kReachZ, iy = (i / kReachZ) % kReachY, ix = i / (kReachZ * kReachY);
        const int vx = x0 + ix, vy = y0 + iy, vz = z0 + iz;
        if (vx >= p.nx || vy >= p.ny || vz >= p.nz) continue;
        const long long v = (long long)vx * plane + vy * p.nz + vz;
        const int c = cnt[v];
        if (c < 2) continue;
        const int cx = ix + r, cy = iy + r, cz = iz + r;   // own place in the halo
        unsigned word = 0;
        int bit = 0;
        for (int b = 1; b < c; b++)
        {
            const int B = idx[b * N + v];
            for (int a = 0; a < b; a++, bit++)
            {
                const unsigned key = pair_code(idx[a * N + v], B);
                unsigned h = (key * 2654435761u) >> 24;
                int probe = 0;
                for (; probe < kReachKeys && key_of[h] != key && key_of[h] != 0u; probe++) h = (h + 1) & (kReachKeys - 1);
                bool hit = false;
                if (probe < kReachKeys && key_of[h] == key)
                    for (int e = first[h]; e < first[h + 1] && !hit; e++)
                    {
                        const unsigned at = place[e];
                        const int dx = (int)(at >> 20) - cx, dy = (int)((at >> 10) & 1023u) - cy, dz = (int)(at & 1023u) - cz;
                        hit = dx * dx + dy * dy + dz * dz < r * r;   // Range - |d| > 0
                    }
                if (hit) word |= 1u << (bit & 31);
                if ((bit & 31) == 31)
                {
                    aa.mask[(long long)(bit >> 5) * N + v] = word;
                    word = 0;
                }
            }
        }
        if (bit & 31) aa.mask[(long long)(bit >> 5) * N + v] = word;
    }
}

// The direct search for the tiles that df_reach_kernel listed (gy, gx: tiles along y and z).  How long a
// voxel searches depends on where it lies, so that the warps fetch 32 voxels at a time.
template <class R>
__global__ void __launch_bounds__(128) df_tiles_kernel(const __grid_constant__ StepParams p, AvgArrays aa, unsigned gy,
                                                        unsigned gx, const uint8_t* __restrict__ cnt,
                                                        const int16_t* __restrict__ idx, const R* __restrict__ val,
                                                        const double* __restrict__ vr)
{
    constexpr unsigned kParts = kReachX * kReachY * kReachZ / 32;
    const unsigned items = aa.tiles[0] * kParts, lane = threadIdx.x & 31u, warps = gridDim.x * (blockDim.x >> 5);
    // a warp's first item is its own number (no tile listed: nothing is fetched), the next ones are counted
    for (unsigned item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < items;)
    {
        const unsigned tile = aa.tiles[2u + item / kParts], i = (item % kParts) * 32u + lane;
        const int x = (int)(tile / (gx * gy) * kReachX + i / (kReachZ * kReachY));
        const int y = (int)(tile / gx % gy * kReachY + i / kReachZ % kReachY);
        const int z = (int)(tile % gx * kReachZ + i % kReachZ);
        if (x < p.nx && y < p.ny && z < p.nz) search_sphere<R>(p, aa, cnt, idx, val, vr, x, y, z);
        __syncwarp();
        item = lane == 0 ? warps + atomicAdd(&aa.tiles[1], 1u) : 0u;
        item = __shfl_sync(0xffffffffu, item, 0);
    }
}

template <class R>
int launch_average_of(const StepParams& p, const AvgArrays& aa, const uint8_t* cnt, const int16_t* idx, const R* val,
                      const double* vr, cudaStream_t s, int* kernels)
{
    df_mark_kernel<R><<<(unsigned)((p.n + 255) / 256), 256, 0, s>>>(p.n, aa.weight_threshold, cnt, idx, val, vr, aa.strong,
                                                                  aa.tiles);
    const dim3 tiles((p.nz + kReachZ - 1) / kReachZ, (p.ny + kReachY - 1) / kReachY, (p.nx + kReachX - 1) / kReachX);
    if (aa.range <= kReachRange && tiles.y <= 65535u && tiles.z <= 65535u)
    {
        df_reach_kernel<R><<<tiles, 256, 0, s>>>(p, aa, cnt, idx, val, vr);
        df_tiles_kernel<R><<<148 * 8, 128, 0, s>>>(p, aa, tiles.y, tiles.x, cnt, idx, val, vr);
        *kernels += 3;
    }
    else
    {
        df_sphere_kernel<R><<<(unsigned)((p.n + 127) / 128), 128, 0, s>>>(p, aa, cnt, idx, val, vr);
        *kernels += 2;
    }
    return (int)cudaGetLastError();
}

}  // namespace

size_t average_tiles(int nx, int ny, int nz)
{
    return (size_t)((nx + kReachX - 1) / kReachX) * ((ny + kReachY - 1) / kReachY) * ((nz + kReachZ - 1) / kReachZ);
}

int launch_average(const StepParams& p, const AvgArrays& aa, const uint8_t* cnt, const int16_t* idx,
                   const void* val, bool fp32, const double* vr, void* stream, int* kernels)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return fp32 ? launch_average_of<float>(p, aa, cnt, idx, static_cast<const float*>(val), vr, s, kernels)
                : launch_average_of<double>(p, aa, cnt, idx, static_cast<const double*>(val), vr, s, kernels);
}

}  // namespace opgpu
