// Where an element of a row-major block goes under a permutation of its axes:
// the block permutation kernel's index arithmetic (host code as well, so that
// the branch for blocks of 2^31 elements and more is tested without one).
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define KV_PERM_HD __host__ __device__ __forceinline__
#else
#define KV_PERM_HD inline
#endif

namespace kvp {

constexpr int kRank = 6;

struct PermMap {
    // strides and lengths of the input's axes, and the output stride of each (0 past the rank)
    unsigned sd[kRank], sh[kRank];
    int64_t od[kRank];
    bool same;  // the identity
};

// shape, perm: [rank]; output axis j is input axis perm[j]
KV_PERM_HD PermMap perm_map(const int64_t *shape, const int64_t *perm, int rank) {
    PermMap m;
    int64_t st = 1;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = kRank - 1; i >= 0; --i) {
        m.sh[i] = i < rank ? (unsigned)shape[i] : 1u;
        m.sd[i] = (unsigned)st;
        m.od[i] = 0;
        st *= m.sh[i];
    }
    m.same = true;
    int64_t ost = 1;
    for (int j = rank - 1; j >= 0; --j) {
        const int ax = (int)perm[j];
        m.same = m.same && ax == j;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int i = 0; i < kRank; ++i)
            if (i == ax) {
                m.od[i] = ost;
                ost *= m.sh[i];
            }
    }
    return m;
}

// output index of input element e; wide: the block has 2^31 elements or more
// (64-bit divisions, by the lengths: strides may not fit 32 bits)
KV_PERM_HD int64_t perm_index(const PermMap &m, int rank, int64_t e, bool wide) {
    if (m.same) return e;
    int64_t dst = 0;
    if (wide) {
        int64_t rem = e;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int i = kRank - 1; i >= 0; --i)
            if (i < rank) {
                dst += (rem % m.sh[i]) * m.od[i];
                rem /= m.sh[i];
            }
    } else {
        unsigned rem = (unsigned)e;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int i = 0; i < kRank; ++i)
            if (i < rank) {
                const unsigned x = rem / m.sd[i];
                rem -= x * m.sd[i];
                dst += x * m.od[i];
            }
    }
    return dst;
}

}  // namespace kvp
