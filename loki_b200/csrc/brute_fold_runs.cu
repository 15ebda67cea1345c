// Brute fold, run form (sm_100a).
//
// Same sums as brute_fold.cu: every bin adds its samples in increasing sample
// order from 0.0f, E and V in one add.rn.f32x2, the bins' sums in shared
// memory. There a warp walks the samples and tests every one for a run start;
// here the unit of work is the run:
//  * lane = segment (32 segments share one frequency's run structure, so all
//    control flow is uniform), warp = one trial frequency and one range of at
//    most kRangeMax bins (more bins are folded as several ranges, each reading
//    only its own samples);
//  * the series is first transposed to [32-segment group][sample][lane] (e, v)
//    pairs, so a sample is one conflict-free 256-byte warp read at any offset;
//  * a rotation's runs have L or L + 1 samples (L = floor(samples per bin)):
//    the plan stores, per rotation, the sample where the range starts and one
//    bit per bin for the longer runs. Two or four consecutive bins' sums and
//    samples are loaded together and added in independent chains (L < 16, a
//    compile-time constant); longer runs go one at a time in steps of 16;
//  * runs cut by the segment's ends are read at full length: the transposed
//    segments have zeros before and after them, and adding +0.0 changes no
//    sum (a sum that starts at +0.0 is never -0.0 in round-to-nearest);
//  * a producer thread streams the samples through a shared-memory ring of
//    bulk copies; the first samples of slot 0 are also copied behind the last
//    slot, so a unit that reads past the end of the ring needs no wrap.
//
// What bounds it: shared memory, 8 bytes per (sample, frequency) for the
// samples -- every frequency reads every sample once -- and 16 per run for its
// sums, at 128 bytes per clock and SM. Measured on B200: the 2^22-sample
// accelerated workload (nbins 64, 755 frequencies, 5-49 samples per run) 1.08
// ms, 83 % of the shared-memory wavefront rate (1.83 ms walking samples, 1.56
// with its launch shape tuned and tensor-memory warps); the 2^21-sample period
// sweep (nbins 128, 3020 frequencies) 3.23 against 6.91; nbins 100 0.41
// against 0.74; 512 bins 0.86 against 3.18; 1024 bins 0.39 against 2.79; 64
// segments of 50 frequencies (nbins 32) 0.023 against 0.056. Series with unit
// variances fold E alone (see pairs_e): 0.60 ms and 76 % of the wavefront rate at
// 64 bins, 1.83 ms and 61 % at 128, where runs of 2 to 24 samples leave their
// sums' 16 bytes and latency to weigh more.
//
// Keeping the sums in registers (the bin loop unrolled, a few runs' code per
// bin) saves the 16 bytes but measured slower: the unrolled code outgrows the
// instruction caches (64 bins per warp: 62 % of the issue slots without an
// instruction, 3.81 ms on the 2^22-sample accelerated workload; 32 bins: 2.00).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "lk_device.cuh"
#include "lk_fold_runs.hpp"
#include "lk_ptx.cuh"

namespace lk {

namespace {

constexpr uint32_t kStageLen = 32;                      // samples per ring stage
constexpr uint32_t kSampleBytes = 32 * sizeof(float2);  // one sample of 32 segments
constexpr uint32_t kStageBytes = kStageLen * kSampleBytes;
constexpr uint32_t kMirror = 32;     // samples copied behind the ring: a unit's reach
constexpr uint32_t kMinSlots = 4;
constexpr uint32_t kMaxSlots = 12;
constexpr uint32_t kRangeMax = 64;   // bins per warp
static_assert(kRangeMax <= 64, "a rotation's longer runs are one 64-bit word");
constexpr uint32_t kChunk = 16;      // run lengths below are compile-time: 2 runs (4 below 8) fit the mirror
constexpr uint32_t kMaxLen = 2048;   // longest run
constexpr uint32_t kMaxWarps = 20;
constexpr size_t kSmemLimit = 227 * 1024;

// Shared memory: ring, mirror, barriers, sums.
constexpr uint32_t ring_bytes(uint32_t slots) { return slots * kStageBytes; }
constexpr uint32_t sums_offset(uint32_t slots) {
    return ring_bytes(slots) + kMirror * kSampleBytes + 2 * kMaxSlots * sizeof(uint64_t);
}
size_t smem_bytes(uint32_t slots, uint32_t warps, uint32_t range) {
    return sums_offset(slots) + static_cast<size_t>(warps) * range * kSampleBytes;
}

// One (bin range, frequency): its rotations are rots[rot0 .. rot0 + nrot).
struct RunItem {
    uint32_t rot0, nrot;
    uint32_t t0;    // first bin group (of 4) of the first rotation
    uint32_t t1;    // bin groups of the last rotation
    uint32_t len;   // L
    uint32_t bins;  // bins of the range
};

struct RunArgs {
    const RunItem* items;  // [nranges][nfreq]
    const uint32_t* rots;  // first sample (padded) of each rotation of a range
    const uint32_t* bits;  // [rotation][wpr] longer-run bits of the range's bins
    const float2* evt;     // [group][nstages * kStageLen][32]
    uint32_t nfreq, nseg, nbins;
    uint32_t range;        // bins per range (a multiple of 4)
    uint32_t wpr;          // words of bits per rotation
    uint32_t nfb;          // frequency blocks per range
    uint32_t warps;
    uint32_t slots;
    uint32_t nstages;
    float* fold;
    uint32_t* status;
    const uint32_t* groups;
    const uint32_t* ngroups;
    // Unit variances (nullptr: every group folds (e, v) pairs): groups of 64
    // segments whose flag is 0 hold ones in V throughout; their pairs are the E
    // of segments l and l + 32, and V's sums are the bins' sample counts.
    const uint32_t* varied;
    const float* counts;   // [nfreq][nbins]
};

__device__ __forceinline__ float2 add2_rn(float2 a, float2 b) {
    uint64_t ra, rb, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(rd));
    return r;
}

extern __shared__ __align__(128) unsigned char fold_smem[];

__device__ __forceinline__ uint64_t* full_bar(const RunArgs& a, uint32_t slot) {
    return reinterpret_cast<uint64_t*>(fold_smem + ring_bytes(a.slots) + kMirror * kSampleBytes) + slot;
}
__device__ __forceinline__ uint64_t* empty_bar(const RunArgs& a, uint32_t slot) {
    return full_bar(a, slot) + kMaxSlots;
}

// A warp's view of the ring: the samples below `have` have landed, the stages
// below `gone` / kStageLen are released.
struct Ring {
    uint32_t have = 0, hslot = 0, hparity = 0;
    uint32_t gone = 0, gslot = 0;

    __device__ __forceinline__ void release(const RunArgs& a, int lane) {
        __syncwarp();
        if (lane == 0) {
            ptx::mbar_arrive(empty_bar(a, gslot));
        }
        gone += kStageLen;
        gslot = gslot + 1 == a.slots ? 0 : gslot + 1;
    }
    // Waits until the samples below q_end have landed (false when a wait gave
    // up); those below q are no longer needed by this warp: the loads of all of
    // them are done, as their sums have been stored (an arrival alone does not
    // wait for loads, see ptx::loads_done).
    __device__ __forceinline__ bool acquire(uint32_t q, uint32_t q_end, const RunArgs& a, int lane) {
#pragma unroll 1
        do {
#pragma unroll 1
            while (gone + kStageLen <= min(q, have)) {
                release(a, lane);
            }
            const bool got =
                ptx::mbar_wait_bounded(full_bar(a, hslot), hparity, a.status,
                                       dev::kStatusWaitTimeout | (have == 0 ? dev::kStatusFirstFull : dev::kStatusFull));
            if (!__all_sync(0xffffffffu, got)) {
                return false;
            }
            have += kStageLen;
            if (++hslot == a.slots) {
                hslot = 0;
                hparity ^= 1u;
            }
        } while (q_end > have);
        return true;
    }
};

// Adds N samples from p to s, in order, then one more when `extra`.
template <int N>
__device__ __forceinline__ float2 add_run(float2 s, const unsigned char* p, bool extra) {
    float2 x[N + 1];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = *reinterpret_cast<const float2*>(p + i * kSampleBytes);
    }
    if (extra) {
        x[N] = *reinterpret_cast<const float2*>(p + N * kSampleBytes);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        s = add2_rn(s, x[i]);
    }
    if (extra) {
        s = add2_rn(s, x[N]);
    }
    return s;
}

// Adds the runs of UB bins, L or L + 1 (bit k of m) samples each, from p to
// the sums at acc, BB bins in flight together.
template <int L, int UB>
__device__ __forceinline__ void add_unit(unsigned char* acc, const unsigned char* p, uint32_t m) {
    constexpr int BB = L <= 4 ? 4 : 2;
#pragma unroll
    for (int k0 = 0; k0 < UB; k0 += BB) {
        float2 s[BB], x[BB][L + 1];
#pragma unroll
        for (int k = 0; k < BB; ++k) {
            s[k] = *reinterpret_cast<const float2*>(acc + (k0 + k) * kSampleBytes);
#pragma unroll
            for (int i = 0; i < L; ++i) {
                x[k][i] = *reinterpret_cast<const float2*>(p + i * kSampleBytes);
            }
            if (m & (1u << (k0 + k))) {
                x[k][L] = *reinterpret_cast<const float2*>(p + L * kSampleBytes);
                p += kSampleBytes;
            }
            p += L * kSampleBytes;
        }
#pragma unroll
        for (int i = 0; i < L; ++i) {
#pragma unroll
            for (int k = 0; k < BB; ++k) {
                s[k] = add2_rn(s[k], x[k][i]);
            }
        }
#pragma unroll
        for (int k = 0; k < BB; ++k) {
            if (m & (1u << (k0 + k))) {
                s[k] = add2_rn(s[k], x[k][L]);
            }
            *reinterpret_cast<float2*>(acc + (k0 + k) * kSampleBytes) = s[k];
        }
    }
}

// Folds one item. Units of UB = 4 bins (L < 8) or 2 (L < 16), L = LF at compile
// time, or of one bin with L = 16 * nfull + LF (UB = 1).
template <int LF, int UB>
__device__ __forceinline__ bool fold_item(unsigned char* sums, Ring& rg, const RunArgs& a, const RunItem& it, int lane) {
    constexpr bool LONG = UB == 1;
    constexpr uint32_t UPW = 32 / UB;  // units per word of bits
    const uint32_t nfull = LONG ? it.len / kChunk : 0;
    const uint32_t rbytes = ring_bytes(a.slots);
    const uint32_t rlen = a.slots * kStageLen;
    // units per rotation (one bin at a time: only the bins there are, so that
    // a rotation's start never lies before a unit that was waited for)
    const uint32_t upr = LONG ? it.bins : (it.bins + UB - 1) / UB;
    const unsigned char* ring = fold_smem + lane * sizeof(float2);
    const uint32_t* rots = a.rots + it.rot0;
    const uint32_t* bits = a.bits + static_cast<size_t>(it.rot0) * a.wpr + min(static_cast<uint32_t>(lane), a.wpr - 1);
    uint32_t nq = __ldg(rots), nm = __ldg(bits);  // of the next rotation
    uint32_t u = it.t0 * (4 / UB);  // the first rotation starts at its first run's group
    for (uint32_t r = 1; r <= it.nrot; ++r) {
        uint32_t q = nq;
        const uint32_t mine = nm;  // lane w: word w of the rotation's bits
        uint32_t off = (q % rlen) * kSampleBytes;
        uint32_t uend = upr;
        if (r < it.nrot) {
            nq = __ldg(rots + r);
            nm = __ldg(bits + static_cast<size_t>(r) * a.wpr);
        } else {
            uend = min(upr, it.t1 * (4 / UB));  // units of the last rotation
        }
        unsigned char* acc = sums + u * UB * kSampleBytes;
        while (u < uend) {
            uint32_t m = __shfl_sync(0xffffffffu, mine, u / UPW) >> (u * UB % 32);
            const uint32_t uw = min(uend, (u / UPW + 1) * UPW);
#pragma unroll 1
            for (; u < uw; ++u) {
                if constexpr (!LONG) {
                    if (q + UB * (LF + 1) > rg.have && !rg.acquire(q, q + UB * (LF + 1), a, lane)) {
                        return false;
                    }
                    add_unit<LF, UB>(acc, ring + off, m);
                    const uint32_t adv = UB * LF + __popc(m & ((1u << UB) - 1));
                    q += adv;
                    off += adv * kSampleBytes;
                } else {
                    // (the chunk before is kept, its samples' sum is in a register and
                    // the adds that used the one before that came first; q starts
                    // kChunk or more into the padding)
                    float2 s = *reinterpret_cast<const float2*>(acc);
#pragma unroll 1
                    for (uint32_t c = 0; c < nfull; ++c) {
                        if (q + kChunk > rg.have && !rg.acquire(q - kChunk, q + kChunk, a, lane)) {
                            return false;
                        }
                        s = add_run<kChunk - 1>(s, ring + off, true);
                        q += kChunk;
                        off += kChunk * kSampleBytes;
                        off = off >= rbytes ? off - rbytes : off;
                    }
                    if (q + kChunk > rg.have && !rg.acquire(q - kChunk, q + kChunk, a, lane)) {
                        return false;
                    }
                    *reinterpret_cast<float2*>(acc) = add_run<LF>(s, ring + off, (m & 1u) != 0);
                    q += LF + (m & 1u);
                    off += (LF + (m & 1u)) * kSampleBytes;
                }
                off = off >= rbytes ? off - rbytes : off;
                acc += UB * kSampleBytes;
                m >>= UB;
            }
        }
        u = 0;
    }
    return true;
}

// fold_item by the run length: 0 .. 15 at compile time, then by its remainder.
template <int C = 0>
__device__ __forceinline__ bool fold_dispatch(uint32_t cls, unsigned char* sums, Ring& rg, const RunArgs& a,
                                              const RunItem& it, int lane) {
    if constexpr (C == 2 * kChunk) {
        return true;
    } else {
        if (cls == C) {
            constexpr int UB = C < 8 ? 4 : (C < static_cast<int>(kChunk) ? 2 : 1);
            return fold_item<C % static_cast<int>(kChunk), UB>(sums, rg, a, it, lane);
        }
        return fold_dispatch<C + 1>(cls, sums, rg, a, it, lane);
    }
}

__global__ void __launch_bounds__((kMaxWarps + 1) * 32, 1) brute_fold_runs_kernel(const __grid_constant__ RunArgs a) {
    if (a.ngroups != nullptr && blockIdx.x * 4u >= *a.ngroups) {
        return;  // uniform: no segment group for this block
    }
    const bool unit = a.varied != nullptr && a.varied[blockIdx.x / 2] == 0;
    if (unit && (blockIdx.x & 1u) != 0) {
        return;  // uniform: folded by the group's other block
    }
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0);
    const int lane = static_cast<int>(threadIdx.x % 32);
    // The highest frequencies (most run starts) first.
    const uint32_t range = blockIdx.y / a.nfb;
    const uint32_t f0 = (a.nfb - 1 - (blockIdx.y - range * a.nfb)) * a.warps;
    const uint32_t nw = min(a.warps, a.nfreq - f0);
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < a.slots; ++s) {
            ptx::mbar_init(full_bar(a, s), 1);
            ptx::mbar_init(empty_bar(a, s), nw);
        }
        ptx::fence_barrier_init();
    }
    __syncthreads();

    if (warp == a.warps) {
        if (lane == 0) {
            const float2* src = a.evt + static_cast<size_t>(blockIdx.x) * a.nstages * (kStageLen * 32);
            uint32_t slot = 0, parity = 1;  // of the use before
            uint32_t k = 0;
            for (; k < a.nstages; ++k) {
                if (k >= a.slots && !ptx::mbar_wait_bounded(empty_bar(a, slot), parity, a.status,
                                                            dev::kStatusWaitTimeout | dev::kStatusEmpty)) {
                    break;
                }
                const float2* p = src + static_cast<size_t>(k) * (kStageLen * 32);
                uint64_t* full = full_bar(a, slot);
                constexpr uint32_t kMirrorBytes = kMirror * kSampleBytes;
                static_assert(kMirrorBytes <= kStageBytes, "the mirror is part of slot 0");
                ptx::mbar_arrive_expect_tx(full, slot == 0 ? kStageBytes + kMirrorBytes : kStageBytes);
                ptx::bulk_load(fold_smem + slot * kStageBytes, p, kStageBytes, full);
                if (slot == 0) {
                    ptx::bulk_load(fold_smem + ring_bytes(a.slots), p, kMirrorBytes, full);
                }
                if (++slot == a.slots) {
                    slot = 0;
                    parity ^= 1u;
                }
            }
            // Stay resident until the last copies have landed (bounded).
            for (uint32_t j = k > a.slots ? k - a.slots : 0; j < k; ++j) {
                ptx::mbar_wait_bounded(full_bar(a, j % a.slots), (j / a.slots) & 1u, a.status,
                                       dev::kStatusWaitTimeout | dev::kStatusDrain);
            }
        }
        return;
    }
    if (warp >= nw) {
        return;
    }
    const uint32_t f = f0 + warp;
    const RunItem it = a.items[static_cast<size_t>(range) * a.nfreq + f];
    unsigned char* sums = fold_smem + sums_offset(a.slots) + static_cast<size_t>(warp) * a.range * kSampleBytes +
                          lane * sizeof(float2);
    for (uint32_t b = 0; b < a.range; ++b) {
        *reinterpret_cast<float2*>(sums + b * kSampleBytes) = make_float2(0.0f, 0.0f);
    }
    Ring rg;
    const uint32_t cls = it.len < kChunk ? it.len : kChunk + it.len % kChunk;
    if (it.nrot > 0 && !fold_dispatch(cls, sums, rg, a, it, lane)) {
        return;
    }
    // The rest of the segment passes unread.
    const uint32_t all = a.nstages * kStageLen;
    if (rg.have < all && !rg.acquire(all, all, a, lane)) {
        return;
    }

    const float2* A = reinterpret_cast<const float2*>(sums);
    const float* cnt = unit ? a.counts + static_cast<size_t>(f) * a.nbins + range * a.range : nullptr;
    for (uint32_t h = 0; h < (unit ? 2u : 1u); ++h) {
        const uint32_t grp = blockIdx.x + h;
        uint32_t seg = grp * 32u + static_cast<uint32_t>(lane);
        bool store = seg < a.nseg;
        if (a.groups != nullptr) {
            const uint32_t g = grp * 4u + static_cast<uint32_t>(lane / 8);
            store = g < *a.ngroups;
            seg = store ? a.groups[g] + static_cast<uint32_t>(lane % 8) : 0u;
        }
        if (!store) {
            continue;
        }
        float* out = a.fold + (static_cast<size_t>(seg) * a.nfreq + f) * 2 * a.nbins + range * a.range;
        auto pair = [&](uint32_t b) {  // bin b's (E, V) of this segment
            const float2 p = A[b * 32];
            return unit ? make_float2(h == 0 ? p.x : p.y, __ldg(cnt + b)) : p;
        };
        if ((a.nbins & 3u) == 0) {  // then ranges start and end on 4 bins
            for (uint32_t b = 0; b < it.bins; b += 4) {
                const float2 p0 = pair(b), p1 = pair(b + 1), p2 = pair(b + 2), p3 = pair(b + 3);
                *reinterpret_cast<float4*>(out + b) = make_float4(p0.x, p1.x, p2.x, p3.x);
                *reinterpret_cast<float4*>(out + a.nbins + b) = make_float4(p0.y, p1.y, p2.y, p3.y);
            }
        } else {
            for (uint32_t b = 0; b < it.bins; ++b) {
                const float2 p = pair(b);
                out[b] = p.x;
                out[a.nbins + b] = p.y;
            }
        }
    }
}

// Segments (rows of seglen samples) to [group][pad + sample][lane] (e, v)
// pairs. Block: 64 samples of one group of 32 segments through a shared tile,
// so reads are along the samples and writes along the lanes. HBM-bound.
constexpr int kTile = 64;
__global__ void __launch_bounds__(256)
    transpose_ev_kernel(const float* __restrict__ e, const float* __restrict__ v, float2* __restrict__ evt,
                        uint32_t nrows, uint32_t seglen, uint32_t pad, uint32_t qlen, bool vec4,
                        const uint32_t* groups, const uint32_t* ngroups, const uint32_t* varied) {
    __shared__ float2 tile[kTile][33];
    const uint32_t tiles = (seglen + kTile - 1) / kTile;
    const uint32_t grp = blockIdx.x / tiles;
    if (varied != nullptr && varied[grp / 2] == 0) {
        return;  // laid out by pair_e_kernel
    }
    if (ngroups != nullptr && grp * 4u >= *ngroups) {
        return;
    }
    const uint32_t s0 = (blockIdx.x - grp * tiles) * kTile;
    const uint32_t j = threadIdx.x / 8, c = threadIdx.x % 8;
    uint32_t row = grp * 32u + j;
    bool have = row < nrows;
    if (groups != nullptr) {
        const uint32_t g = grp * 4u + j / 8;
        have = g < *ngroups;
        row = have ? groups[g] + j % 8 : 0u;
    }
    if (have) {
        const float* pe = e + static_cast<size_t>(row) * seglen;
        const float* pv = v + static_cast<size_t>(row) * seglen;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t i = 4 * c + 32 * h;
            if (s0 + i < seglen) {  // seglen is a multiple of 4
                float4 x, y;
                if (vec4) {
                    x = __ldg(reinterpret_cast<const float4*>(pe + s0 + i));
                    y = __ldg(reinterpret_cast<const float4*>(pv + s0 + i));
                } else {
                    x = make_float4(__ldg(pe + s0 + i), __ldg(pe + s0 + i + 1), __ldg(pe + s0 + i + 2),
                                    __ldg(pe + s0 + i + 3));
                    y = make_float4(__ldg(pv + s0 + i), __ldg(pv + s0 + i + 1), __ldg(pv + s0 + i + 2),
                                    __ldg(pv + s0 + i + 3));
                }
                tile[i][j] = make_float2(x.x, y.x);
                tile[i + 1][j] = make_float2(x.y, y.y);
                tile[i + 2][j] = make_float2(x.z, y.z);
                tile[i + 3][j] = make_float2(x.w, y.w);
            }
        }
    }
    __syncthreads();
    const uint32_t n = min(static_cast<uint32_t>(kTile), seglen - s0);
    float2* out = evt + (static_cast<size_t>(grp) * qlen + pad + s0) * 32;
    for (uint32_t i = threadIdx.x; i < n * 32; i += 256) {
        out[i] = tile[i / 32][i % 32];
    }
}

// Groups of 64 segments to [group][pad + sample][lane] pairs of the E of segments
// lane and lane + 32, as far as their V is 1.0f throughout; a group with any
// other V is flagged in varied (zero on entry) and left to transpose_ev_kernel.
__global__ void __launch_bounds__(256)
    pair_e_kernel(const float* __restrict__ e, const float* __restrict__ v, float2* __restrict__ evt, uint32_t nrows,
                  uint32_t seglen, uint32_t pad, uint32_t qlen, bool vec4, const uint32_t* groups,
                  const uint32_t* ngroups, uint32_t* varied) {
    __shared__ float tile[kTile][65];
    const uint32_t tiles = (seglen + kTile - 1) / kTile;
    const uint32_t g64 = blockIdx.x / tiles;
    if (ngroups != nullptr && g64 * 8u >= *ngroups) {
        return;
    }
    const uint32_t s0 = (blockIdx.x - g64 * tiles) * kTile;
    const uint32_t c = threadIdx.x % 8;
    bool ones = true;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t j = threadIdx.x / 8 + 32 * half;
        uint32_t row = g64 * 64u + j;
        bool have = row < nrows;
        if (groups != nullptr) {
            const uint32_t g = g64 * 8u + j / 8;
            have = g < *ngroups;
            row = have ? groups[g] + j % 8 : 0u;
        }
        const float* pe = e + static_cast<size_t>(row) * seglen;
        const float* pv = v + static_cast<size_t>(row) * seglen;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t i = 4 * c + 32 * h;
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (have && s0 + i < seglen) {  // seglen is a multiple of 4
                float4 y;
                if (vec4) {
                    x = __ldg(reinterpret_cast<const float4*>(pe + s0 + i));
                    y = __ldg(reinterpret_cast<const float4*>(pv + s0 + i));
                } else {
                    x = make_float4(__ldg(pe + s0 + i), __ldg(pe + s0 + i + 1), __ldg(pe + s0 + i + 2),
                                    __ldg(pe + s0 + i + 3));
                    y = make_float4(__ldg(pv + s0 + i), __ldg(pv + s0 + i + 1), __ldg(pv + s0 + i + 2),
                                    __ldg(pv + s0 + i + 3));
                }
                ones = ones && y.x == 1.0f && y.y == 1.0f && y.z == 1.0f && y.w == 1.0f;
            }
            tile[i][j] = x.x;
            tile[i + 1][j] = x.y;
            tile[i + 2][j] = x.z;
            tile[i + 3][j] = x.w;
        }
    }
    if (__syncthreads_or(!ones)) {
        if (threadIdx.x == 0) {
            varied[g64] = 1;
        }
        return;
    }
    const uint32_t n = min(static_cast<uint32_t>(kTile), seglen - s0);
    float2* out = evt + (static_cast<size_t>(2 * g64) * qlen + pad + s0) * 32;
    for (uint32_t i = threadIdx.x; i < n * 32; i += 256) {
        out[i] = make_float2(tile[i / 32][i % 32], tile[i / 32][i % 32 + 32]);
    }
}

struct RunTables {
    bool ok = false;
    uint32_t nranges = 1, range = 0, pad = 0, nstages = 0;
    std::vector<RunItem> items;
    std::vector<uint32_t> rots;
    std::vector<uint32_t> bits;
    std::vector<float> counts;  // samples of each frequency's bins in one segment
    uint32_t wpr = 1;
};

// The kernel's tables, or ok = false where it does not apply.
RunTables build_tables(const std::vector<double>& freqs, uint64_t segment_len, uint32_t nbins, double tsamp,
                       double t_ref) {
    const auto nfreq = static_cast<uint32_t>(freqs.size());
    const auto seglen = static_cast<uint32_t>(segment_len);
    RunTables tb;
    tb.nranges = (nbins + kRangeMax - 1) / kRangeMax;
    tb.range = ((nbins + tb.nranges - 1) / tb.nranges + 3) / 4 * 4;
    tb.nranges = (nbins + tb.range - 1) / tb.range;
    tb.wpr = (tb.range + 31) / 32;
    if (segment_len > (1u << 30) || segment_len % 4 != 0) {
        return tb;
    }
    // Of one frequency: the run length L and, range after range, its rotations
    // (first samples without the padding).
    struct Freq {
        bool ok = false;
        uint32_t len = 0;
        std::vector<RunItem> items;
        std::vector<int64_t> rots;
        std::vector<uint32_t> bits;
    };
    // A thread's scratch: the runs, and the rotations of each range so far.
    struct Scratch {
        FoldRuns runs;
        std::vector<uint32_t> cnt;
        std::vector<std::vector<int64_t>> rots;
        std::vector<std::vector<uint64_t>> longer;
    };
    std::vector<Freq> fr(nfreq);
    tb.counts.resize(static_cast<size_t>(nfreq) * nbins);
    const uint32_t ng = tb.range / 4;
    parallel_for<Scratch>(nfreq, fold_run_evaluations(freqs, tsamp, nbins, segment_len), [&](uint64_t f, Scratch& sc) {
        fold_runs(freqs[f], segment_len, nbins, tsamp, t_ref, sc.runs);
        const auto& st = sc.runs.start;
        const auto& bn = sc.runs.bin;
        const size_t n = st.size();
        auto len_of = [&](size_t j) { return (j + 1 < n ? st[j + 1] : seglen) - st[j]; };
        uint32_t lo = 0xffffffffu, hi = 0;
        for (size_t j = 1; j + 1 < n; ++j) {
            const uint32_t len = st[j + 1] - st[j];
            lo = std::min(lo, len);
            hi = std::max(hi, len);
        }
        bool seq = true;  // bins step by one
        size_t rotations = 1, last_start = 0;
        for (size_t j = 1; j < n; ++j) {
            if (bn[j] <= bn[j - 1]) {
                seq &= bn[j] == 0 && bn[j - 1] == nbins - 1;
                last_start = j;
                ++rotations;
            } else {
                seq &= bn[j] == bn[j - 1] + 1u;
            }
        }
        const uint32_t c0 = len_of(0), c1 = len_of(n - 1);
        uint32_t len = 0;
        int64_t first = 0;  // where the first run, made up to at least L samples, starts
        if (!seq) {
            // Bins are skipped: every run is one sample and every other bin
            // none (L = 0). Frequencies near the sampling rate, whose
            // rotations hold a sample or two, are left to the other forms.
            if ((n > 2 && hi > 1) || c0 > 1 || c1 > 1 || rotations > seglen / 4 + 1) {
                return;
            }
        } else {
            if (n <= 2) {
                lo = hi = std::max(c0, c1);
            }
            if (hi > lo + 1 || c0 > lo + 1 || c1 > lo + 1 || lo + 1 > kMaxLen) {
                return;
            }
            len = lo;
            first = n > 1 ? static_cast<int64_t>(st[1]) - std::max(c0, lo) : 0;
        }
        sc.cnt.assign(nbins, 0);
        sc.rots.resize(tb.nranges);
        sc.longer.resize(tb.nranges);
        Freq x;
        x.len = len;
        x.items.resize(tb.nranges);
        for (uint32_t rg = 0; rg < tb.nranges; ++rg) {
            sc.rots[rg].clear();
            sc.longer[rg].clear();
            x.items[rg] = RunItem{};
            x.items[rg].len = len;
            x.items[rg].bins = std::min(tb.range, nbins - rg * tb.range);
        }
        for (size_t k = 0; k < n;) {  // one rotation of one range
            const uint32_t rg = bn[k] / tb.range;
            const uint32_t rg0 = rg * tb.range, rg_end = rg0 + tb.range;
            RunItem& it = x.items[rg];
            int64_t pos = st[k];
            if (seq && k == 0) {
                // the first run, from the first bin of its group
                pos = first - static_cast<int64_t>((bn[k] - rg0) % 4) * len;
                it.t0 = (bn[k] - rg0) / 4;
            }
            uint64_t longer = 0;  // bit per bin: a run of more than L samples
            uint32_t b = bn[k], next = b;
            do {
                b = next;
                const uint32_t cur = (k + 1 < n ? st[k + 1] : seglen) - st[k];
                sc.cnt[b] += cur;
                longer |= static_cast<uint64_t>(cur > len) << (b - rg0);
                next = ++k < n ? bn[k] : 0;
            } while (next > b && next < rg_end);
            it.t1 = seq && k > last_start ? (b - rg0) / 4 + 1 : ng;
            sc.rots[rg].push_back(pos);
            sc.longer[rg].push_back(longer);
        }
        std::copy(sc.cnt.begin(), sc.cnt.end(), tb.counts.begin() + f * nbins);
        for (uint32_t rg = 0; rg < tb.nranges; ++rg) {
            x.items[rg].nrot = static_cast<uint32_t>(sc.rots[rg].size());
            x.rots.insert(x.rots.end(), sc.rots[rg].begin(), sc.rots[rg].end());
            for (const uint64_t w : sc.longer[rg]) {
                x.bits.push_back(static_cast<uint32_t>(w));
                if (tb.wpr == 2) {
                    x.bits.push_back(static_cast<uint32_t>(w >> 32));
                }
            }
        }
        x.ok = true;
        fr[f] = std::move(x);
    });
    uint32_t lmax = 0;
    size_t total = 0;
    for (const Freq& x : fr) {
        if (!x.ok) {
            return tb;
        }
        lmax = std::max(lmax, x.len + 1);
        total += x.rots.size();
    }
    // A group of 4 bins reaches up to 4 runs before the segment's first
    // sample and past its last one.
    const uint32_t reach = 4 * lmax + kChunk;
    tb.pad = (reach + kStageLen - 1) / kStageLen * kStageLen;
    tb.nstages = (tb.pad + seglen + reach + kStageLen - 1) / kStageLen;
    if (total > 0x7fffffffULL) {
        return tb;
    }
    tb.items.resize(static_cast<size_t>(tb.nranges) * nfreq);
    tb.rots.reserve(std::max<size_t>(total, 1));
    tb.bits.reserve(std::max<size_t>(total, 1) * tb.wpr);
    for (uint32_t f = 0; f < nfreq; ++f) {
        uint32_t at = static_cast<uint32_t>(tb.rots.size());
        for (uint32_t rg = 0; rg < tb.nranges; ++rg) {
            RunItem& it = tb.items[static_cast<size_t>(rg) * nfreq + f];
            it = fr[f].items[rg];
            it.rot0 = at;
            at += it.nrot;
        }
        for (const int64_t pos : fr[f].rots) {
            tb.rots.push_back(static_cast<uint32_t>(pos + tb.pad));
        }
        tb.bits.insert(tb.bits.end(), fr[f].bits.begin(), fr[f].bits.end());
    }
    tb.ok = true;
    return tb;
}

}  // namespace

namespace {

uint64_t transposed_bytes(uint64_t max_rows, uint32_t nstages) {
    return (max_rows + 31) / 32 * nstages * kStageBytes;
}

// Whether the run form is taken for a call's segments. Speed: every block streams
// the padding too, four runs and more on both sides. Against the form that walks
// samples (times as fast, unit variances / others), 2^20 and 2^22 samples, 48 and
// 96 frequencies, 16 to 128 bins: segments of 2048 samples and more padded to
// less than twice their length 1.1 to 4.3 / 1.0 to 2.5, to 4.5 times 0.7 to 1.0;
// segments of 256 to 1024 samples padded to at most 1.5 times 1.0 to 2.3 / 0.82 to
// 1.7 (below 1 where bins are skipped or hold 9 and more samples), to 3.7 and
// 10 times 0.6 to 1.0 / 0.35 to 0.7; of 64 and 16 samples, padded to 2 and 6
// times and more, 0.8 to 1.2 / 0.7 to 1.2. Memory: 32 segments' worth for each group even
// where the call has fewer (2 to 4.5 times as fast there all the same), so at
// most twice the series' (e, v) pairs or 1 GiB.
bool run_form_pays(uint64_t segment_len, uint32_t nstages, uint64_t max_rows) {
    const uint64_t padded = static_cast<uint64_t>(nstages) * kStageLen;
    const uint64_t pairs = max_rows * segment_len * sizeof(float2);
    return (segment_len >= 2048 ? padded <= 2 * segment_len : 2 * padded <= 3 * segment_len) &&
           transposed_bytes(max_rows, nstages) <= std::max<uint64_t>(2 * pairs, 1ull << 30);
}

}  // namespace

bool run_form_applies(const std::vector<double>& freqs, uint64_t segment_len, uint64_t nbins, double tsamp,
                      double t_ref, uint64_t max_rows, uint64_t* bytes) {
    const RunTables tb = build_tables(freqs, segment_len, static_cast<uint32_t>(nbins), tsamp, t_ref);
    *bytes = tb.ok ? transposed_bytes(max_rows, tb.nstages) : 0;
    return tb.ok && run_form_pays(segment_len, tb.nstages, max_rows);
}

RunFold::RunFold(const std::vector<double>& freqs, uint64_t segment_len, uint64_t nbins, double tsamp, double t_ref,
                 uint64_t max_rows)
    : m_nfreq(static_cast<uint32_t>(freqs.size())),
      m_nbins(static_cast<uint32_t>(nbins)),
      m_seglen(static_cast<uint32_t>(segment_len)),
      m_max_rows(max_rows) {
    const RunTables tb = build_tables(freqs, segment_len, m_nbins, tsamp, t_ref);
    if (!tb.ok || !run_form_pays(segment_len, tb.nstages, max_rows)) {
        return;
    }
    m_nranges = tb.nranges;
    m_range = tb.range;
    m_pad = tb.pad;
    m_nstages = tb.nstages;
    m_items.alloc(tb.items.size() * sizeof(RunItem));
    LK_CUDA(cudaMemcpy(m_items.ptr, tb.items.data(), m_items.bytes, cudaMemcpyHostToDevice));
    m_rots.alloc(tb.rots.size() * sizeof(uint32_t));
    LK_CUDA(cudaMemcpy(m_rots.ptr, tb.rots.data(), m_rots.bytes, cudaMemcpyHostToDevice));
    m_bits.alloc(tb.bits.size() * sizeof(uint32_t));
    LK_CUDA(cudaMemcpy(m_bits.ptr, tb.bits.data(), m_bits.bytes, cudaMemcpyHostToDevice));
    m_wpr = tb.wpr;
    m_counts.alloc(tb.counts.size() * sizeof(float));
    LK_CUDA(cudaMemcpy(m_counts.ptr, tb.counts.data(), m_counts.bytes, cudaMemcpyHostToDevice));
    m_ok = true;
}

bool run_fold_replay(const std::vector<double>& freqs, uint64_t segment_len, uint64_t nbins, double tsamp,
                     double t_ref, const float* ts, float* fold) {
    const auto nfreq = static_cast<uint32_t>(freqs.size());
    const RunTables tb = build_tables(freqs, segment_len, static_cast<uint32_t>(nbins), tsamp, t_ref);
    if (!tb.ok) {
        return false;
    }
    const uint64_t qlen = static_cast<uint64_t>(tb.nstages) * kStageLen;
    std::vector<float> x(qlen, 0.0F);
    std::copy(ts, ts + segment_len, x.begin() + tb.pad);
    const uint32_t ng = (tb.range + 3) / 4;
    std::fill(fold, fold + nfreq * nbins, 0.0F);
    for (uint32_t rg = 0; rg < tb.nranges; ++rg) {
        const uint32_t nb = std::min<uint32_t>(tb.range, static_cast<uint32_t>(nbins) - rg * tb.range);
        for (uint32_t f = 0; f < nfreq; ++f) {
            const RunItem& it = tb.items[static_cast<size_t>(rg) * nfreq + f];
            std::vector<float> acc(4 * ng, 0.0F);
            uint64_t released = 0;  // samples below this are gone from the ring
            for (uint32_t r = 0; r < it.nrot; ++r) {
                uint64_t q = tb.rots[it.rot0 + r];
                const uint32_t* rot = &tb.bits[static_cast<size_t>(it.rot0 + r) * tb.wpr];
                // the kernel's units
                const uint32_t ub = it.len < 8 ? 4 : (it.len < kChunk ? 2 : 1);
                const uint32_t upr = (it.bins + ub - 1) / ub;
                const uint32_t uend = r + 1 < it.nrot ? upr : std::min(upr, it.t1 * (4 / ub));
                for (uint32_t u = r == 0 ? it.t0 * (4 / ub) : 0; u < uend; ++u) {
                    const uint64_t end = q + (ub == 1 ? it.len + kChunk : ub * (it.len + 1));
                    require(q >= released && (ub > 1 || q >= kChunk) && end <= qlen,
                            "run fold table: unit outside the segment");
                    released = q / kStageLen * kStageLen;
                    for (uint32_t b = u * ub; b < (u + 1) * ub; ++b) {
                        const uint32_t n = it.len + ((rot[b / 32] >> (b & 31)) & 1U);
                        for (uint32_t i = 0; i < n; ++i, ++q) {
                            acc[b] += x.at(q);
                        }
                    }
                }
            }
            std::copy(acc.begin(), acc.begin() + nb, fold + f * nbins + rg * tb.range);
        }
    }
    return true;
}

uint32_t RunFold::marker_stages() { return 32; }

namespace {

uint32_t sm_count() {
    int dev = 0, nsm = 148;
    LK_CUDA(cudaGetDevice(&dev));
    LK_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    return static_cast<uint32_t>(nsm);
}

}  // namespace

uint32_t RunFold::max_warps() const {
    const size_t fixed = smem_bytes(kMinSlots, 0, 0);
    return static_cast<uint32_t>(std::min<size_t>((kSmemLimit - fixed) / (m_range * kSampleBytes), kMaxWarps));
}

// A wave of blocks takes time in proportion to about 4 + its warps (2^22-sample
// accelerated workload, nbins 64: 0.181 ms a wave with 5 warps, 0.191 with 6,
// 0.270 with 11; 64 segments of 50 frequencies, one wave: 0.023 ms with 5,
// 0.029 with 10, 0.050 with 20). Series with unit variances take half the
// blocks of others, and which it will be is not known here: the warps with the
// smallest product of the two costs (waves x (4 + warps)). Over 25 plans (32 to
// 256 bins, 2^16 to 2^22 samples) that is on average 1.1 % above the best warps
// with unit variances and 3.0 % with others; the smallest cost with unit
// variances alone measured 1.9 and 7.1 %. The fewest warps that give one wave
// win over that when they save series with other variances a fifth of their
// cost at no more than 1.6 times the cost of the rest, as one wave leaves the
// check out too: 128 segments, 336 frequencies of 32 bins 0.056 ms for both with
// 10 warps, 0.052 and 0.077 with 5.
uint32_t RunFold::default_warps(uint64_t nseg) const {
    const uint32_t nsm = sm_count();
    struct Shape {
        uint32_t warps;  // 0, none: more blocks than a launch takes
        uint64_t unit, varied;
    };
    Shape best{0, ~0u, ~0u}, one{0, ~0u, ~0u};
    const uint32_t wmax = max_warps();
    for (uint32_t c = std::min(wmax, 4u); c <= wmax; ++c) {
        const uint64_t per_group = blocks_per_group(c);
        auto cost = [&](uint64_t groups) { return (groups * per_group + nsm - 1) / nsm * (4 + c); };
        Shape s{c, 0, cost((nseg + 31) / 32)};
        s.unit = pairs_e(nseg, c) ? cost((nseg + 63) / 64) : s.varied;
        if (per_group > 65535) {
            continue;
        }
        if (one.warps == 0 && s.varied == 4 + c) {
            one = s;
        }
        if (best.warps == 0 || s.unit * s.varied < best.unit * best.varied) {
            best = s;
        }
    }
    return one.warps != 0 && 10 * one.varied <= 8 * best.varied && 10 * one.unit <= 16 * best.unit ? one.warps
                                                                                                   : best.warps;
}

// Series whose variances are all 1.0f (white noise, the usual input) are checked
// for it on every call and folded with E alone, two segments a lane: V's sums
// are then the sample counts of the plan, exactly what adding ones gives below
// 2^24. That halves the fold: 2^22-sample accelerated search 0.59 ms against
// 1.08, 2^21-sample period sweep at 128 bins 1.81 against 3.24. One wave of
// blocks would take the same time with half the groups, so the check and its
// launches are left out there.
bool RunFold::pairs_e(uint64_t nrows, uint32_t warps) const {
    return nrows > 32 && m_seglen <= (1u << 24) && (nrows + 31) / 32 * blocks_per_group(warps) > sm_count();
}

void RunFold::reserve() {
    if (m_evt.ptr != nullptr) {
        return;
    }
    // the series, then the flags of the groups of 64
    m_evt.alloc(transposed_bytes(m_max_rows, m_nstages) + (m_max_rows + 63) / 64 * sizeof(uint32_t));
    m_varied = reinterpret_cast<uint32_t*>(m_evt.as<unsigned char>() + transposed_bytes(m_max_rows, m_nstages));
    // the zeros before and after each segment stay; the samples between them
    // are written by every call, on any stream (the tables' copies have landed
    // after the wait too)
    LK_CUDA(cudaMemsetAsync(m_evt.ptr, 0, m_evt.bytes, nullptr));
    LK_CUDA(cudaStreamSynchronize(nullptr));
}

void RunFold::transpose(const float* d_e, const float* d_v, uint64_t nrows, uint32_t warps, const uint32_t* groups,
                        const uint32_t* ngroups, cudaStream_t s) {
    const uint64_t ngrp = (nrows + 31) / 32;
    const uint64_t qlen = static_cast<uint64_t>(m_nstages) * kStageLen;
    const uint64_t tiles = (m_seglen + kTile - 1) / kTile;
    require(ngrp * tiles <= 0x7fffffffULL && nrows <= m_max_rows, "BruteFold: too many segments");
    const bool vec4 = (reinterpret_cast<uintptr_t>(d_e) % 16 == 0) && (reinterpret_cast<uintptr_t>(d_v) % 16 == 0);
    m_unit = pairs_e(nrows, warps);
    m_rows = nrows;
    const uint64_t g64 = (nrows + 63) / 64;
    if (m_unit) {
        LK_CUDA(cudaMemsetAsync(m_varied, 0, g64 * sizeof(uint32_t), s));
        pair_e_kernel<<<static_cast<unsigned>(g64 * tiles), 256, 0, s>>>(
            d_e, d_v, m_evt.as<float2>(), static_cast<uint32_t>(nrows), m_seglen, m_pad, static_cast<uint32_t>(qlen),
            vec4, groups, ngroups, m_varied);
        LK_CUDA(cudaGetLastError());
    }
    transpose_ev_kernel<<<static_cast<unsigned>(ngrp * tiles), 256, 0, s>>>(d_e, d_v, m_evt.as<float2>(), static_cast<uint32_t>(nrows), m_seglen,
                                             m_pad, static_cast<uint32_t>(qlen), vec4, groups, ngroups,
                                             m_unit ? m_varied : nullptr);
    LK_CUDA(cudaGetLastError());
}

void RunFold::unit_groups(uint64_t* checked, uint64_t* varied, cudaStream_t s) const {
    std::vector<uint32_t> flags(m_unit ? (m_rows + 63) / 64 : 0);
    if (!flags.empty()) {
        LK_CUDA(cudaMemcpyAsync(flags.data(), m_varied, flags.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        LK_CUDA(cudaStreamSynchronize(s));
    }
    *checked = flags.size();
    *varied = static_cast<uint64_t>(std::count_if(flags.begin(), flags.end(), [](uint32_t x) { return x != 0; }));
}

void RunFold::fold(float* d_fold, uint64_t nrows, uint32_t warps, const uint32_t* groups,
                   const uint32_t* ngroups, uint32_t* d_status, cudaStream_t s) const {
    RunArgs a{};
    a.items = m_items.as<RunItem>();
    a.rots = m_rots.as<uint32_t>();
    a.bits = m_bits.as<uint32_t>();
    a.evt = m_evt.as<float2>();
    a.nfreq = m_nfreq;
    a.nseg = static_cast<uint32_t>(nrows);
    a.nbins = m_nbins;
    a.range = m_range;
    a.wpr = m_wpr;
    a.warps = warps;
    a.nfb = (m_nfreq + warps - 1) / warps;
    a.slots = kMinSlots;
    while (a.slots < kMaxSlots && smem_bytes(a.slots + 1, warps, m_range) <= kSmemLimit) {
        ++a.slots;
    }
    a.nstages = m_nstages;
    a.fold = d_fold;
    a.status = d_status;
    a.groups = groups;
    a.ngroups = ngroups;
    a.varied = m_unit ? m_varied : nullptr;
    a.counts = m_counts.as<float>();
    const uint64_t gy = static_cast<uint64_t>(a.nfb) * m_nranges;
    require(gy <= 65535, "BruteFold: too many frequencies for the launch grid");
    dim3 grid(static_cast<unsigned>((nrows + 31) / 32), static_cast<unsigned>(gy));
    const size_t smem = smem_bytes(a.slots, warps, m_range);
    LK_CUDA(cudaFuncSetAttribute(brute_fold_runs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    brute_fold_runs_kernel<<<grid, (warps + 1) * 32, smem, s>>>(a);
    LK_CUDA(cudaGetLastError());
}

}  // namespace lk
