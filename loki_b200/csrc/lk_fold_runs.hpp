// Run form of the brute fold (brute_fold_runs.cu): host tables and launch.
#pragma once

#include <cstdint>
#include <vector>

#include "lk_host.hpp"
#include "lk_kernels.hpp"

namespace lk {

// The runs of one trial frequency over one segment, in sample order: the first
// sample and the bin of each run of equal bin.
struct FoldRuns {
    std::vector<uint32_t> start;
    std::vector<uint16_t> bin;
};

// The runs of one frequency.
void fold_runs(double freq, uint64_t segment_len, uint64_t nbins, double tsamp, double t_ref, FoldRuns& out);

// Host replay of the run form's tables over one segment of one row (fold:
// [nfreq][nbins]), with the kernel's reads checked against the padded segment;
// false where the form does not apply.
bool run_fold_replay(const std::vector<double>& freqs, uint64_t segment_len, uint64_t nbins, double tsamp,
                     double t_ref, const float* ts, float* fold);

// Whether the run form is the default for calls of up to max_rows segments;
// bytes: of its transposed series.
bool run_form_applies(const std::vector<double>& freqs, uint64_t segment_len, uint64_t nbins, double tsamp,
                      double t_ref, uint64_t max_rows, uint64_t* bytes);

class RunFold {
public:
    // Builds the tables; ok() is false when a frequency's runs do not have
    // the form the kernel takes, or where it does not pay (brute_fold_runs.cu).
    // max_rows: most segments of a call.
    RunFold(const std::vector<double>& freqs, uint64_t segment_len, uint64_t nbins, double tsamp, double t_ref,
            uint64_t max_rows);
    bool ok() const { return m_ok; }
    // Consumer warps per block the kernel allows, and the default for a fold
    // of nseg segments.
    uint32_t max_warps() const;
    uint32_t default_warps(uint64_t nseg) const;
    uint64_t blocks_per_group(uint32_t warps) const {
        return static_cast<uint64_t>(m_nranges) * ((m_nfreq + warps - 1) / warps);
    }
    // Ring depth that names this form in a launch shape (its real depth
    // follows from the shared memory the sums leave).
    static uint32_t marker_stages();
    // Allocates and clears the buffers of max_rows segments (on the first call
    // only; they live as long as the object).
    void reserve();
    // Transposes nrows segments into [group of 32][sample][32 lanes] (e, v)
    // pairs, or groups of 64 with unit variances into pairs of their E, for a
    // fold() of `warps` warps. groups / ngroups: the segment-group table
    // (nullptr: all rows in order).
    void transpose(const float* d_e, const float* d_v, uint64_t nrows, uint32_t warps, const uint32_t* groups,
                   const uint32_t* ngroups, cudaStream_t s);
    void fold(float* d_fold, uint64_t nrows, uint32_t warps, const uint32_t* groups,
              const uint32_t* ngroups, uint32_t* d_status, cudaStream_t s) const;
    // Groups of 64 segments whose variances the last transpose() checked (0: not
    // checked, both rows folded) and those found with other variances than 1
    // (synchronises s).
    void unit_groups(uint64_t* checked, uint64_t* varied, cudaStream_t s) const;
    uint64_t device_bytes() const {
        return m_items.bytes + m_rots.bytes + m_bits.bytes + m_counts.bytes + m_evt.bytes;
    }

private:
    bool pairs_e(uint64_t nrows, uint32_t warps) const;
    bool m_ok = false;
    bool m_unit = false;  // the transposed rows were checked for unit variances
    uint64_t m_rows = 0;  // of the last transpose()
    uint32_t m_nfreq, m_nbins, m_seglen;
    uint32_t m_nranges = 1, m_range = 0;  // bin ranges per frequency, bins per range
    uint32_t m_pad = 0;                   // zero samples before each segment
    uint32_t m_nstages = 0;               // stages of one padded segment
    DeviceBuffer m_items, m_rots, m_bits, m_counts, m_evt;
    uint32_t* m_varied = nullptr;         // inside m_evt: flags of the groups of 64 segments
    uint32_t m_wpr = 1;
    uint64_t m_max_rows;
};

}  // namespace lk
