// CASToR list-mode events on the GPU: prompt histogramming and scatter
// injection (the reference's Timber package, Python/Timber/Datafile.py).
//
//  * histogram_kernel: one thread per event.  Crystal IDs -> (crystal, ring)
//    pairs and TOF sign as ParseCASToRIDs (Coincidence.py:97-159), sinogram
//    cell from the LOR and slice tables, TOF bin as ExportPrompts
//    (Datafile.py:86-113); counts are 32-bit atomics, reduced to the
//    reference's wrapping uint16 at the end.  The randoms and normalisation
//    sinograms keep the value of the last event (file order) of each cell,
//    as the reference's per-event assignment does: atomicMax of the event
//    number, then a pass over the cells writes the winners' values.
//  * tile_*: the same by tiles of cells in shared memory, wherever these hold
//    the problem (up to 2^31 events).
//  * inject_*: InjectScatters (Datafile.py:117-240): events outside the TOF
//    range or the tables are dropped, the others get a scatter rate inserted
//    after their correction factors; the kept events keep file order
//    (block counts, one scan, ordered writes).
#include <cmath>

#include "common.cuh"

namespace {

using namespace sss;

struct Parsed {
    int d1, r1, d2, r2;  // crystal (unshifted, d1 < d2) and ring of each side
    float tof;           // ps, sign for the (r1, r2) order
};

__device__ __forceinline__ uint32_t load_u32(const unsigned char* rec, int off)
{
    return *reinterpret_cast<const uint32_t*>(rec + off);
}

__device__ __forceinline__ float load_f32(const unsigned char* rec, int off)
{
    return *reinterpret_cast<const float*>(rec + off);
}

// ParseCASToRIDs (Coincidence.py:97-159) for the event at rec.
__device__ __forceinline__ Parsed parse_event(const unsigned char* rec, const sss_listmode_layout& L, int ncr,
                                              int shift)
{
    const uint32_t a = load_u32(rec, L.id_offset), b = load_u32(rec, L.id_offset + 4);
    const float tof = load_f32(rec, L.tof_offset);
    const uint32_t id1 = a < b ? a : b, id2 = a < b ? b : a;
    const float tof_t = a < b ? tof : -tof;
    Parsed P;
    const uint32_t q1 = id1 / (uint32_t)ncr, q2 = id2 / (uint32_t)ncr;
    const int c1 = (int)(id1 - q1 * (uint32_t)ncr), c2 = (int)(id2 - q2 * (uint32_t)ncr);
    P.d1 = c1 < c2 ? c1 : c2;
    P.d2 = c1 < c2 ? c2 : c1;
    int s1 = c1 - shift, s2 = c2 - shift;
    if (s1 < 0) s1 += ncr;
    if (s2 < 0) s2 += ncr;
    if (s1 < s2) {
        P.r1 = (int)q1;
        P.r2 = (int)q2;
        P.tof = tof_t;
    } else {
        P.r1 = (int)q2;
        P.r2 = (int)q1;
        P.tof = -tof_t;
    }
    return P;
}

// Sinogram cell of an event: -1 = skipped as the reference skips it, -2 =
// outside the tables (the reference raises IndexError).
__device__ __forceinline__ long long event_cell(const Parsed& P, const sss_sino_map& M)
{
    const int i1 = P.d1 / M.mash, i2 = P.d2 / M.mash;
    if (i1 >= M.nd_lor || i2 >= M.nd_lor || P.r1 >= M.nr_table || P.r2 >= M.nr_table) return -2;
    const int ang = M.lor[2 * ((long long)i1 * M.nd_lor + i2)];
    const int rad = M.lor[2 * ((long long)i1 * M.nd_lor + i2) + 1];
    const int sino = M.slices[(long long)P.r1 * M.nr_table + P.r2];
    if (sino == -1 || rad == -1 || ang == -1) return -1;
    if (rad < 0 || rad >= M.nrad || ang < 0 || ang >= M.nang || sino < 0 || sino >= M.nslices) return -2;
    return ((long long)rad * M.nang + ang) * M.nslices + sino;
}

// TOF bin as the reference computes it in FP64 (Datafile.py:103-110); -1 = the
// TOF is outside the range, -2 = inside it but in no bin (the upper end).  The
// FP64 pipe runs at about 1/70 of the FP32 rate, so the two FP64 divisions are
// left to events near a bin edge: t below differs from the exact quotient by a
// few FP32 roundings of tof_bins at most, well within kBinEdge * tof_bins.  (A
// NaN TOF or quotient falls to the FP64 form, too.)
constexpr float kBinEdge = 2e-6f;

struct TofRule {  // FP32 forms of the map's range and bins; scale 0: FP64 only
    float range, scale, bins, edge;
    double width;  // of a bin
};

TofRule tof_rule(const sss_sino_map& M)
{
    TofRule R;
    R.range = (float)M.tof_range;
    R.bins = (float)M.tof_bins;
    R.edge = kBinEdge * R.bins;
    R.width = (2.0 * M.tof_range) / M.tof_bins;
    R.scale = R.range > 1e-30f && R.range < 1e30f ? R.bins / (2.0f * R.range) : 0.f;
    return R;
}

__device__ __forceinline__ int tof_bin(float tof, const TofRule& R, const sss_sino_map& M)
{
    if (R.scale > 0.f) {
        const float t32 = (tof + R.range) * R.scale;
        if (t32 < -R.edge || t32 > R.bins + R.edge) return -1;
        if (fabsf(t32 - rintf(t32)) > R.edge) return (int)t32;
    }
    const double x = (double)tof;
    if (fabs(x) > M.tof_range) return -1;
    const double t = (x + M.tof_range) / R.width;
    if (t < 0.0 || t >= (double)M.tof_bins) return -2;
    return (int)t;
}

// A cell's randoms value from event[0] of its last event: the reference's
// (float)(event[0] * duration / tof_bins) in FP64 (Datafile.py:95-99).  The
// product with c = duration / tof_bins is formed in pairs of FP32 numbers
// (Dekker's products with fused multiply-adds; event[0] as two 16-bit parts, c as
// 48 bits), off by less than 2^-45 of itself; where both ends of an interval of
// 2^-42 of it round to the same float, that float is the FP64 form's.  Where
// duration and c have few bits (whole seconds), every step is exact and the
// interval a point, so that ties between two floats need no second look.  Else,
// and outside FP32's comfortable range, the FP64 form itself.
struct RandomsRule {
    double duration;
    int tof_bins;
    float hi, lo;  // duration / tof_bins; hi 0: FP64 only
    float slack;   // relative half width of the interval
};

RandomsRule randoms_rule(double duration, int tof_bins)
{
    RandomsRule Q;
    Q.duration = duration;
    Q.tof_bins = tof_bins;
    const double c = duration / tof_bins;
    const bool fits = c > 1e-15 && c < 1e25;
    Q.hi = fits ? (float)c : 0.f;
    Q.lo = fits ? (float)(c - (double)Q.hi) : 0.f;
    // v has at most `bits` significant bits
    auto short_value = [](double v, int bits) {
        int e;
        const double m = ldexp(frexp(v, &e), bits);
        return m == floor(m);
    };
    const bool exact = fits && tof_bins < (1 << 24) && short_value(c, 16) && short_value(duration, 21) &&
                       c * tof_bins == duration;
    Q.slack = exact ? 0.f : 0x1p-42f;
    return Q;
}

__device__ __forceinline__ float randoms_value(uint32_t first, const RandomsRule& Q)
{
    if (Q.hi > 0.f) {
        const float th = (float)(first & 0xffff0000u), tl = (float)(first & 0xffffu);
        const float p1 = __fmul_rn(th, Q.hi), e1 = __fmaf_rn(th, Q.hi, -p1);
        const float p2 = __fmul_rn(tl, Q.hi), e2 = __fmaf_rn(tl, Q.hi, -p2);
        const float s = __fadd_rn(p1, p2), e3 = __fsub_rn(p2, __fsub_rn(s, p1));  // p1 = 0 or p1 > p2
        const float low = __fmaf_rn(__fadd_rn(th, tl), Q.lo, __fadd_rn(e3, __fadd_rn(e1, e2)));
        const float eta = __fmul_rn(s, Q.slack);
        const float a = __fadd_rn(s, __fsub_rn(low, eta)), b = __fadd_rn(s, __fadd_rn(low, eta));
        if (a == b) return a;  // event[0] = 0: 0
    }
    return (float)(((double)first * Q.duration) / Q.tof_bins);
}

__global__ void histogram_kernel(const unsigned char* __restrict__ ev, long long n, sss_listmode_layout L,
                                 sss_sino_map M, TofRule R, unsigned int* __restrict__ counts,
                                 unsigned long long* __restrict__ last, int32_t* status)
{
    const int ncr = M.nd_lor * M.mash;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
         e += (long long)gridDim.x * blockDim.x) {
        const Parsed P = parse_event(ev + e * L.record_bytes, L, ncr, M.shift);
        const long long cell = event_cell(P, M);
        if (cell == -2) {
            raise_error(status, kErrEvent);
            continue;
        }
        if (cell < 0) continue;
        if (last) atomicMax(last + cell, (unsigned long long)(e + 1));
        const int bin = tof_bin(P.tof, R, M);
        if (bin < 0) continue;
        atomicAdd(counts + cell * M.tof_bins + bin, 1u);
    }
}

__global__ void histogram_finish_kernel(const unsigned int* __restrict__ counts, long long n,
                                        uint16_t* __restrict__ prompts)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        prompts[i] = (uint16_t)(counts[i] & 0xffffu);  // numpy uint16 += 1 wraps
}

// One thread per cell: the cell's last event (numbered from 1 by the
// histogram pass, 0 = none) gives its randoms and normalisation values,
// event[0] * scan_duration / TOF_bins and event[1] (Datafile.py:95-99).  The
// cells are read in order and only the winning events at random: cheaper
// than parsing every event again to find the winners.
__global__ void last_values_kernel(const unsigned char* __restrict__ ev, long long n, sss_listmode_layout L,
                                   long long ncell, RandomsRule Q, const unsigned long long* __restrict__ last,
                                   float* __restrict__ randoms, float* __restrict__ norm)
{
    for (long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x; cell < ncell;
         cell += (long long)gridDim.x * blockDim.x) {
        const unsigned long long e1 = last[cell];
        if (e1 == 0 || e1 > (unsigned long long)n) continue;
        const unsigned char* rec = ev + (long long)(e1 - 1) * L.record_bytes;
        if (randoms) randoms[cell] = randoms_value(load_u32(rec, 0), Q);
        if (norm) norm[cell] = load_f32(rec, 4);
    }
}

// ---- The histogram by tiles of cells: the direct form's two atomics an event go
// to random sectors of memory far beyond L2 and back (its last-value pass reads
// the winners' records at random again), so the events are first put in order of
// their tile, and a block takes a tile's counters in shared memory.
//   tile_count_kernel    key of each event, and its place in its tile
//   tile_scan_kernel     first record of each tile
//   tile_scatter_kernel  the events' records by tile
//   tile_kernel          a tile's counts, last events and output
// 50 million events into 58 million cells of 6 bins: 0.9 + 0.95 + 0.6 ms, where
// the direct form took 3.95 (histogram_kernel), 1.27 (last values), 0.33 and 0.4
// ms (zeroes).  tile_count_kernel waits for its returning atomics,
// tile_scatter_kernel for its 16-byte writes to 22000 tiles.  Shared memory of 72
// KB a tile: three blocks a SM hide one another's latencies.

constexpr int kTileBytes = 72 * 1024;  // shared memory of a tile: three blocks a SM
constexpr int kTileThreads = 512;
constexpr uint32_t kNoKey = 0xffffffffu;

struct TileShape {
    long long ncell;
    int codes;         // TOF bins + 1: the last is "no bin" (the event counts as the cell's last only)
    unsigned cells;    // of a tile, a multiple of 32
    unsigned tiles;
    bool want;         // last events' values wanted
};

// false: the form does not hold the problem (keys beyond 32 bits, a cell's
// counters beyond the shared memory)
bool tile_shape(long long n, const sss_sino_map& M, bool want, TileShape& S)
{
    S.ncell = (long long)M.nrad * M.nang * M.nslices;
    S.want = want;
    const long long per = kTileBytes / (4ll * M.tof_bins + (want ? 4 : 0)) / 32 * 32;
    if (per < 32) return false;
    S.codes = M.tof_bins + 1;
    if (n > 0x7ffffff0ll || S.ncell > 0xfffffff0ll / S.codes) return false;
    S.cells = (unsigned)per;
    S.tiles = (unsigned)((S.ncell + per - 1) / per);
    return true;
}

struct TileWork {
    unsigned *counts, *first;  // [tiles], [tiles + 1]
    uint2* key_place;          // [n]
    void* records;             // [n]: uint4 (key in the tile, event, its first two words), or the key only
};

size_t tile_work(void* base, long long n, const TileShape& S, TileWork& W)
{
    size_t at = 0;
    auto take = [&](size_t bytes) {
        char* p = (char*)base + at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    W.counts = (unsigned*)take(4 * (size_t)S.tiles);
    W.first = (unsigned*)take(4 * ((size_t)S.tiles + 1));
    W.key_place = (uint2*)take(8 * (size_t)n);
    W.records = take((S.want ? 16 : 4) * (size_t)n);
    return at;
}

// Event j of a thread.  Blocks take the events in file order, and in the same
// order in both passes: a tile's consecutive records are then written close
// together in time and leave L2 as whole sectors.
constexpr int kTileItems = 4, kTileBlock = 256 * kTileItems;

__device__ __forceinline__ long long tile_event(int j)
{
    return (long long)blockIdx.x * kTileBlock + j * 256 + threadIdx.x;
}

__global__ void __launch_bounds__(256) tile_count_kernel(const unsigned char* __restrict__ ev, long long n,
                                                         sss_listmode_layout L, sss_sino_map M, TofRule R, TileShape S,
                                                         unsigned* counts, uint2* __restrict__ key_place, int32_t* status)
{
    const int ncr = M.nd_lor * M.mash;
    uint2 kp[kTileItems];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < kTileItems; ++j) {
        const long long e = tile_event(j);
        kp[j] = make_uint2(kNoKey, 0);
        if (e >= n) continue;
        const Parsed P = parse_event(ev + e * L.record_bytes, L, ncr, M.shift);
        const long long cell = event_cell(P, M);
        bad |= cell == -2;
        const int bin = tof_bin(P.tof, R, M);
        if (cell >= 0 && (bin >= 0 || S.want)) kp[j].x = (unsigned)cell * S.codes + (bin >= 0 ? bin : M.tof_bins);
    }
#pragma unroll
    for (int j = 0; j < kTileItems; ++j)
        if (kp[j].x != kNoKey) kp[j].y = atomicAdd(counts + kp[j].x / (S.cells * (unsigned)S.codes), 1u);
#pragma unroll
    for (int j = 0; j < kTileItems; ++j)
        if (tile_event(j) < n) key_place[tile_event(j)] = kp[j];
    if (bad) raise_error(status, kErrEvent);
}

__global__ void __launch_bounds__(1024) tile_scan_kernel(const unsigned* __restrict__ counts, unsigned tiles,
                                                         unsigned* __restrict__ first)
{
    __shared__ unsigned sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned base = 0;
    for (unsigned t0 = 0; t0 < tiles; t0 += 4096) {  // four tiles a thread
        unsigned c[4], s = 0;
        const unsigned t = t0 + 4 * threadIdx.x;
        for (int k = 0; k < 4; ++k) s += c[k] = t + k < tiles ? counts[t + k] : 0;
        unsigned v = s;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) sums[warp] = v;
        __syncthreads();
        if (warp == 0) {
            unsigned w = sums[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += u;
            }
            sums[lane] = w;
        }
        __syncthreads();
        unsigned run = base + v - s + (warp ? sums[warp - 1] : 0);
        for (int k = 0; k < 4; ++k) {
            if (t + k < tiles) first[t + k] = run;
            run += c[k];
        }
        base += sums[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) first[tiles] = base;
}

__global__ void __launch_bounds__(256) tile_scatter_kernel(const unsigned char* __restrict__ ev, long long n,
                                                           int record_bytes, TileShape S,
                                                           const uint2* __restrict__ key_place,
                                                           const unsigned* __restrict__ first, void* __restrict__ records)
{
    const unsigned span = S.cells * (unsigned)S.codes;
#pragma unroll
    for (int j = 0; j < kTileItems; ++j) {
        const long long e = tile_event(j);
        if (e >= n) continue;
        const uint2 kp = key_place[e];
        if (kp.x == kNoKey) continue;
        const unsigned tile = kp.x / span, at = first[tile] + kp.y;
        const unsigned key = kp.x - tile * span;
        if (S.want) {
            const unsigned char* rec = ev + e * record_bytes;
            reinterpret_cast<uint4*>(records)[at] = make_uint4(key, (unsigned)e, load_u32(rec, 0), load_u32(rec, 4));
        } else {
            reinterpret_cast<unsigned*>(records)[at] = key;
        }
    }
}

__global__ void __launch_bounds__(kTileThreads) tile_kernel(TileShape S, const unsigned* __restrict__ first,
                                                            const void* __restrict__ records, RandomsRule Q,
                                                            uint16_t* __restrict__ prompts, float* __restrict__ randoms,
                                                            float* __restrict__ norm)
{
    extern __shared__ __align__(16) unsigned tile_counts[];  // [cells][bins], then [cells] last events
    const int bins = S.codes - 1;
    const unsigned tile = blockIdx.x, ncounts = S.cells * bins, nwords = ncounts + (S.want ? S.cells : 0);
    unsigned* const last = tile_counts + ncounts;
    for (unsigned i = threadIdx.x; i < nwords / 4; i += kTileThreads)  // cells is a multiple of 32
        reinterpret_cast<uint4*>(tile_counts)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const unsigned r0 = first[tile], r1 = first[tile + 1];
    const uint4* const full = reinterpret_cast<const uint4*>(records);
    // key and event of a record; four records' loads are in flight at a time
    auto record = [&](unsigned r) {
        if (r >= r1) return make_uint2(kNoKey, 0);
        return S.want ? *reinterpret_cast<const uint2*>(full + r)
                      : make_uint2(reinterpret_cast<const unsigned*>(records)[r], 0);
    };
    for (unsigned r = r0 + threadIdx.x; r < r1; r += 4 * kTileThreads) {
        uint2 ke[4];
        for (int k = 0; k < 4; ++k) ke[k] = record(r + k * kTileThreads);
        for (int k = 0; k < 4; ++k) {
            if (ke[k].x == kNoKey) break;
            const unsigned cell = ke[k].x / (unsigned)S.codes, code = ke[k].x - cell * S.codes;
            if (code < (unsigned)bins) atomicAdd(tile_counts + cell * bins + code, 1u);
            if (S.want) atomicMax(last + cell, ke[k].y + 1);
        }
    }
    __syncthreads();
    if (S.want) {  // the last events' records take their numbers' place, marked by the top bit
        for (unsigned r = r0 + threadIdx.x; r < r1; r += 4 * kTileThreads) {
            uint2 ke[4];
            for (int k = 0; k < 4; ++k) ke[k] = record(r + k * kTileThreads);
            for (int k = 0; k < 4; ++k) {
                if (ke[k].x == kNoKey) break;
                const unsigned cell = ke[k].x / (unsigned)S.codes;
                if (last[cell] == ke[k].y + 1) last[cell] = 0x80000000u | (r + k * kTileThreads);
            }
        }
        __syncthreads();
    }
    const long long cell0 = (long long)tile * S.cells;
    const unsigned cells = (unsigned)min((long long)S.cells, S.ncell - cell0), outs = cells * bins;
    uint16_t* const out = prompts + cell0 * bins;  // numpy uint16 += 1 wraps
    const bool words = (uintptr_t)out % 8 == 0;
    for (unsigned i = threadIdx.x; words && i < outs / 4; i += kTileThreads) {
        const uint4 c = reinterpret_cast<const uint4*>(tile_counts)[i];
        reinterpret_cast<uint2*>(out)[i] = make_uint2((c.x & 0xffffu) | c.y << 16, (c.z & 0xffffu) | c.w << 16);
    }
    for (unsigned i = (words ? outs / 4 * 4 : 0) + threadIdx.x; i < outs; i += kTileThreads)
        out[i] = (uint16_t)(tile_counts[i] & 0xffffu);
    if (!S.want) return;
    for (unsigned c = threadIdx.x; c < cells; c += kTileThreads) {
        const unsigned v = last[c];
        uint2 value = make_uint2(0, __float_as_uint(1.0f));
        if (v) value = reinterpret_cast<const uint2*>(full + (v & 0x7fffffffu))[1];
        if (randoms) randoms[cell0 + c] = v ? randoms_value(value.x, Q) : 0.f;
        if (norm) norm[cell0 + c] = __uint_as_float(value.y);
    }
}

// ------------------------------------------------------------------ injection

// The scatter values are read at random: 64 bytes filled from memory instead of
// the 128 that a miss brings by default (1.71 instead of 2.89 GB a 20 million
// events; 1.5% of the call).
__device__ __forceinline__ float load_scatter(const float* p)
{
    float v;
    asm("ld.global.L2::64B.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

constexpr int kInjectThreads = 256, kInjectItems = 4, kInjectBlock = kInjectThreads * kInjectItems;

__device__ __forceinline__ bool inject_keep(const unsigned char* rec, const sss_listmode_layout& L,
                                            const sss_sino_map& M, const TofRule& R, const float* scat, const float* factor,
                                            float& rate, bool& bad)
{
    const Parsed P = parse_event(rec, L, M.nd_lor * M.mash, M.shift);
    const int bin = tof_bin(P.tof, R, M);
    if (bin == -1) return false;  // :207-208, before the tables
    const long long cell = event_cell(P, M);
    if (cell == -2) {
        bad = true;
        return false;
    }
    if (cell < 0 || bin < 0) return false;
    const long long ncell = (long long)M.nrad * M.nang * M.nslices;
    rate = __fmul_rn(factor[bin], load_scatter(scat + bin * ncell + cell));  // :229 in float32
    return true;
}

// Event j of a thread: a block's events in rounds of kInjectThreads, in file order.
__device__ __forceinline__ long long inject_event(int j)
{
    return (long long)blockIdx.x * kInjectBlock + j * kInjectThreads + threadIdx.x;
}

__global__ void __launch_bounds__(kInjectThreads) inject_count_kernel(
    const unsigned char* __restrict__ ev, long long n, sss_listmode_layout L, sss_sino_map M, TofRule R,
    const float* __restrict__ scat, const float* __restrict__ factor, unsigned int* __restrict__ block_counts,
    int32_t* status)
{
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    bool bad = false;
    int c = 0;
#pragma unroll
    for (int j = 0; j < kInjectItems; ++j) {
        const long long e = inject_event(j);
        float rate;
        c += e < n && inject_keep(ev + e * L.record_bytes, L, M, R, scat, factor, rate, bad);
    }
    if (bad) raise_error(status, kErrEvent);
    c = __reduce_add_sync(0xffffffffu, c);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) block_counts[blockIdx.x] = (unsigned int)total;
}

// Exclusive scan of the block counts in one block (counts are < 2^32 total
// per block; offsets are 64-bit).
__global__ void __launch_bounds__(1024) inject_scan_kernel(const unsigned int* __restrict__ counts, long long nb,
                                                           unsigned long long* __restrict__ offsets,
                                                           unsigned long long* __restrict__ total)
{
    __shared__ unsigned long long part[1024];
    const long long per = (nb + 1023) / 1024;
    const long long lo = threadIdx.x * per, hi = min(nb, lo + per);
    unsigned long long s = 0;
    for (long long i = lo; i < hi; ++i) s += counts[i];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned long long v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    unsigned long long run = part[threadIdx.x] - s;
    for (long long i = lo; i < hi; ++i) {
        offsets[i] = run;
        run += counts[i];
    }
    if (threadIdx.x == 1023) *total = part[1023];
}

// Bound by memory: 19 million of 20 million events read their scatter value at
// random from 1.4 GB, 2.2 GB in all in 0.6 ms.  Four events a thread shorten the
// scan of the block counts from 72 to 17 us; gathering the output rows for
// coalesced stores was slower (0.76 ms).
__global__ void __launch_bounds__(kInjectThreads) inject_write_kernel(
    const unsigned char* __restrict__ ev, long long n, sss_listmode_layout L, sss_sino_map M, TofRule R,
    const float* __restrict__ scat, const float* __restrict__ factor,
    const unsigned long long* __restrict__ offsets, unsigned char* __restrict__ out, int out_bytes)
{
    constexpr int kWarps = kInjectThreads / 32;
    __shared__ int sums[kInjectItems * kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float rate[kInjectItems];
    unsigned ballot[kInjectItems];
#pragma unroll
    for (int j = 0; j < kInjectItems; ++j) {
        const long long e = inject_event(j);
        bool bad = false;
        rate[j] = 0.f;
        const bool keep = e < n && inject_keep(ev + e * L.record_bytes, L, M, R, scat, factor, rate[j], bad);
        ballot[j] = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) sums[j * kWarps + warp] = __popc(ballot[j]);
    }
    __syncthreads();
    if (warp == 0) {  // 32 sums, in file order
        const int own = sums[lane];
        int s = own;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += v;
        }
        sums[lane] = s;
    }
    __syncthreads();
    const int head = L.scatter_offset / 4, words = L.record_bytes / 4;
    unsigned char* const block_out = out + offsets[blockIdx.x] * (unsigned long long)out_bytes;
#pragma unroll
    for (int j = 0; j < kInjectItems; ++j) {
        if (!(ballot[j] >> lane & 1u)) continue;
        const int at = sums[j * kWarps + warp] - __popc(ballot[j]) + __popc(ballot[j] & ((1u << lane) - 1u));
        const uint32_t* src = reinterpret_cast<const uint32_t*>(ev + inject_event(j) * L.record_bytes);
        uint32_t* d = reinterpret_cast<uint32_t*>(block_out + (long long)at * out_bytes);
        for (int i = 0; i < head; ++i) d[i] = src[i];
        d[head] = __float_as_uint(rate[j]);
        for (int i = head; i < words; ++i) d[i + 1] = src[i];
    }
}
static_assert(kInjectItems * kInjectThreads / 32 == 32, "one warp scans the sums");

int check_layout(const sss_listmode_layout* L, const sss_sino_map* M, const char* who)
{
    if (!L || !M || !M->lor || !M->slices)
        return sss_set_error(SSS_ERR_INVALID, "%s: bad argument", who);
    if (L->record_bytes < 12 || L->record_bytes % 4 || L->id_offset % 4 || L->tof_offset % 4 ||
        L->id_offset < 0 || L->id_offset + 8 > L->record_bytes || L->tof_offset < 0 ||
        L->tof_offset + 4 > L->record_bytes || L->scatter_offset % 4 || L->scatter_offset < 0 ||
        L->scatter_offset > L->record_bytes)
        return sss_set_error(SSS_ERR_INVALID, "%s: event layout must be whole, 4-byte aligned fields", who);
    if (M->nd_lor < 1 || M->mash < 1 || M->nr_table < 1 || M->nrad < 1 || M->nang < 1 || M->nslices < 1 ||
        M->tof_bins < 1 || !(M->tof_range > 0.0))
        return sss_set_error(SSS_ERR_INVALID, "%s: bad sinogram map", who);
    return SSS_OK;
}

unsigned grid_for(long long n, int threads)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long want = (n + threads - 1) / threads, cap = (long long)sms * 16;
    return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

}  // namespace

extern "C" int sss_histogram_prompts(const void* events, int64_t n_events, const sss_listmode_layout* layout,
                                     const sss_sino_map* map, uint32_t* counts, unsigned long long* last,
                                     int32_t* status, void* stream)
{
    int rc = check_layout(layout, map, "sss_histogram_prompts");
    if (rc) return rc;
    if (n_events < 0 || (n_events > 0 && !events) || !counts)
        return sss_set_error(SSS_ERR_INVALID, "sss_histogram_prompts: bad argument");
    if (n_events == 0) return SSS_OK;
    histogram_kernel<<<grid_for(n_events, 256), 256, 0, (cudaStream_t)stream>>>(
        (const unsigned char*)events, n_events, *layout, *map, tof_rule(*map), counts, last, status);
    return sss_check_launch("histogram_kernel");
}

extern "C" int sss_histogram_finish(const void* events, int64_t n_events, const sss_listmode_layout* layout,
                                    const sss_sino_map* map, const uint32_t* counts,
                                    const unsigned long long* last, double duration, uint16_t* prompts,
                                    float* randoms, float* norm, void* stream)
{
    int rc = check_layout(layout, map, "sss_histogram_finish");
    if (rc) return rc;
    if (!counts || !prompts || ((randoms || norm) && !last) || n_events < 0 || (n_events > 0 && !events))
        return sss_set_error(SSS_ERR_INVALID, "sss_histogram_finish: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
    const long long ncell = (long long)map->nrad * map->nang * map->nslices;
    const long long nbins = ncell * map->tof_bins;
    histogram_finish_kernel<<<grid_for(nbins, 256), 256, 0, st>>>(counts, nbins, prompts);
    if ((rc = sss_check_launch("histogram_finish_kernel"))) return rc;
    if ((randoms || norm) && n_events > 0) {
        last_values_kernel<<<grid_for(ncell, 256), 256, 0, st>>>((const unsigned char*)events, n_events, *layout,
                                                                  ncell, randoms_rule(duration, map->tof_bins),
                                                                  last, randoms, norm);
        return sss_check_launch("last_values_kernel");
    }
    return SSS_OK;
}

extern "C" size_t sss_histogram_tiled_workspace_size(int64_t n_events, const sss_sino_map* map, int32_t want_values)
{
    if (n_events < 0 || !map || map->nrad < 1 || map->nang < 1 || map->nslices < 1 || map->tof_bins < 1) return 0;
    TileShape S;
    TileWork W;
    if (!tile_shape(n_events, *map, want_values != 0, S)) return 0;
    return tile_work(nullptr, n_events, S, W);
}

extern "C" int sss_histogram_tiled(const void* events, int64_t n_events, const sss_listmode_layout* layout,
                                   const sss_sino_map* map, double duration, uint16_t* prompts, float* randoms,
                                   float* norm, void* workspace, size_t workspace_bytes, int32_t* status, void* stream)
{
    int rc = check_layout(layout, map, "sss_histogram_tiled");
    if (rc) return rc;
    TileShape S;
    TileWork W;
    if (n_events < 0 || (n_events > 0 && !events) || !prompts || !status)
        return sss_set_error(SSS_ERR_INVALID, "sss_histogram_tiled: bad argument");
    if (!tile_shape(n_events, *map, randoms || norm, S))
        return sss_set_error(SSS_ERR_INVALID, "sss_histogram_tiled: more events, cells or bins than the tiles hold");
    if (!workspace || (uintptr_t)workspace % 16 || workspace_bytes < tile_work(workspace, n_events, S, W))
        return sss_set_error(SSS_ERR_WORKSPACE, "sss_histogram_tiled: workspace too small or not 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned char* ev = (const unsigned char*)events;
    if (cudaMemsetAsync(W.counts, 0, 4 * (size_t)S.tiles, st) != cudaSuccess)
        return sss_set_error(SSS_ERR_CUDA, "sss_histogram_tiled: memset failed");
    const unsigned blocks = (unsigned)((n_events + kTileBlock - 1) / kTileBlock);
    if (n_events > 0) {
        tile_count_kernel<<<blocks, 256, 0, st>>>(ev, n_events, *layout, *map, tof_rule(*map), S, W.counts, W.key_place,
                                                                   status);
        if ((rc = sss_check_launch("tile_count_kernel"))) return rc;
    }
    tile_scan_kernel<<<1, 1024, 0, st>>>(W.counts, S.tiles, W.first);
    if ((rc = sss_check_launch("tile_scan_kernel"))) return rc;
    if (n_events > 0) {
        tile_scatter_kernel<<<blocks, 256, 0, st>>>(ev, n_events, layout->record_bytes, S, W.key_place,
                                                                     W.first, W.records);
        if ((rc = sss_check_launch("tile_scatter_kernel"))) return rc;
    }
    const size_t smem = (size_t)S.cells * (4 * (S.codes - 1) + (S.want ? 4 : 0));
    cudaFuncSetAttribute(tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileBytes);
    tile_kernel<<<S.tiles, kTileThreads, smem, st>>>(S, W.first, W.records, randoms_rule(duration, map->tof_bins), prompts, randoms, norm);
    return sss_check_launch("tile_kernel");
}

extern "C" size_t sss_inject_workspace_size(int64_t n_events)
{
    const long long nb = (n_events + kInjectBlock - 1) / kInjectBlock;
    return (size_t)(((nb * 4 + 255) / 256) * 256 + ((nb * 8 + 255) / 256) * 256 + 256);
}

extern "C" int sss_inject_scatters(const void* events, int64_t n_events, const sss_listmode_layout* layout,
                                   const sss_sino_map* map, const float* scatters, const float* factor,
                                   void* out_events, unsigned long long* out_count, void* workspace,
                                   size_t workspace_bytes, int32_t* status, void* stream)
{
    int rc = check_layout(layout, map, "sss_inject_scatters");
    if (rc) return rc;
    if (n_events < 0 || (n_events > 0 && (!events || !out_events)) || !scatters || !factor || !out_count ||
        !workspace || workspace_bytes < sss_inject_workspace_size(n_events))
        return sss_set_error(SSS_ERR_INVALID, "sss_inject_scatters: bad argument or workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    if (n_events == 0) {
        if (cudaMemsetAsync(out_count, 0, sizeof(unsigned long long), st) != cudaSuccess)
            return sss_set_error(SSS_ERR_CUDA, "sss_inject_scatters: memset failed");
        return SSS_OK;
    }
    const long long nb = (n_events + kInjectBlock - 1) / kInjectBlock;
    if (nb > 0x7fffffffLL) return sss_set_error(SSS_ERR_INVALID, "sss_inject_scatters: too many events");
    char* ws = (char*)workspace;
    unsigned int* counts = (unsigned int*)ws;
    unsigned long long* offsets = (unsigned long long*)(ws + ((nb * 4 + 255) / 256) * 256);
    const unsigned char* ev = (const unsigned char*)events;
    inject_count_kernel<<<(unsigned)nb, kInjectThreads, 0, st>>>(ev, n_events, *layout, *map, tof_rule(*map), scatters, factor,
                                                                  counts, status);
    if ((rc = sss_check_launch("inject_count_kernel"))) return rc;
    inject_scan_kernel<<<1, 1024, 0, st>>>(counts, nb, offsets, out_count);
    if ((rc = sss_check_launch("inject_scan_kernel"))) return rc;
    inject_write_kernel<<<(unsigned)nb, kInjectThreads, 0, st>>>(ev, n_events, *layout, *map, tof_rule(*map), scatters, factor,
                                                                  offsets, (unsigned char*)out_events,
                                                                  layout->record_bytes + 4);
    return sss_check_launch("inject_write_kernel");
}
