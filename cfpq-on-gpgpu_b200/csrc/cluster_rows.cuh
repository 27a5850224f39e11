// Which rows of the matrices and deltas are not empty, as every CTA of the small
// closure's cluster (kernel_cluster.cu) holds it in its own shared memory, and who
// writes what when.  Plain integer code: the kernel runs it, and so does a
// simulation of the cluster on the CPU under random schedules.
//
// Three buffers of delta masks and new-bit counts take turns.  In iteration it a
// CTA reads buffer it % 3, writes (its own copy and, over the cluster, every other
// CTA's) go to buffer (it + 1) % 3, and it sets its own buffer (it + 2) % 3 to
// zero, which nobody else touches before the next cluster barrier.  What a CTA
// reads between two barriers is therefore the same in all of them, however far one
// of them is ahead: a CTA that has begun the next iteration writes to a buffer that
// a CTA still deciding about this one does not read.
//
// The rows of the current matrices have one buffer only, so no other CTA writes
// there: each CTA folds the delta masks that it reads in an iteration into its own
// copy at the iteration's start.  Folding once more changes nothing, so readers
// take the copy together with the delta mask about to be folded, at any time.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CFPQ_HD __host__ __device__ __forceinline__
#else
#define CFPQ_HD inline
#endif

namespace cfpq {

struct ClusterRows {
    static constexpr uint32_t kMats = 32;
    uint64_t *delta;    // [3][nm][T]
    uint64_t *current;  // [nm][T]
    uint32_t *count;    // [3][kMats]
    uint32_t nm, T;

    static CFPQ_HD uint32_t read_buffer(uint32_t it) { return it % 3; }
    static CFPQ_HD uint32_t write_buffer(uint32_t it) { return (it + 1) % 3; }
    static CFPQ_HD uint32_t zero_buffer(uint32_t it) { return (it + 2) % 3; }

    CFPQ_HD uint64_t *delta_rows(uint32_t buf, uint32_t m) const { return delta + ((size_t)buf * nm + m) * T; }

    // Start of iteration it, the CTA's threads together.
    CFPQ_HD void open(uint32_t it, uint32_t tid, uint32_t threads) const {
        for (uint32_t i = tid; i < nm * T; i += threads) {
            delta_rows(zero_buffer(it), 0)[i] = 0;
            current[i] |= delta_rows(read_buffer(it), 0)[i];
        }
        for (uint32_t i = tid; i < kMats; i += threads) count[zero_buffer(it) * kMats + i] = 0;
    }
    // Rows lo, hi (the two halves of word w) of matrix m with `bits` new bits,
    // into buffer buf of every copy: or32(p, v) and add32(p, v) do it for the words
    // that p is in this copy.
    template <class Or, class Add>
    CFPQ_HD void publish(uint32_t buf, uint32_t m, uint32_t w, uint32_t lo, uint32_t hi, uint32_t bits, Or or32,
                         Add add32) const {
        uint32_t *const d = reinterpret_cast<uint32_t *>(delta_rows(buf, m) + w);
        if (lo) or32(d, lo);
        if (hi) or32(d + 1, hi);
        add32(count + buf * kMats + m, bits);
    }
    // Rows of word w that matrix m has after the iteration that wrote buffer buf
    // (until that buffer is zeroed, two iterations on).
    CFPQ_HD uint64_t rows(uint32_t buf, uint32_t m, uint32_t w) const {
        return current[m * T + w] | delta_rows(buf, m)[w];
    }
};

}  // namespace cfpq
