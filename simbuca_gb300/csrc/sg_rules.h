// sg_rules.h -- small rules of the kernels that hold for every size, in plain C++ so that
// they can be checked on the host as well.
#pragma once

#ifdef __CUDACC__
#define SG_HD __host__ __device__ __forceinline__
#else
#define SG_HD inline
#endif

// Frame coordinate (x = y = z) of padding ion g of a cloud: far from every real ion.
SG_HD float sg_pad_frame(int g) { return 1.0e4f + (float)g; }
// Lanes past a cloud's padded end in a 128-ion leaf, on the j side and on the i side of a
// leaf pair: elsewhere than any padding ion, for any cloud size, and than each other.
SG_HD float sg_leaf_fill(bool i_side) { return i_side ? -3.0e4f : -2.0e4f; }

// Whether a close pair of padded indices i, j enters the ions' lists: two different real
// ions (of a cloud whose real ions end at `end`).  Only real ions' lists are emptied again,
// and indices past the padded end are another cloud's or none.
SG_HD bool sg_lists_pair(int i, int j, int end) { return i != j && i < end && j < end; }

// Whether a counter that only rises by one has reached `target`, both modulo 2^32: the
// difference of the two stays far below 2^31, the counts of a long launch do not (a barrier
// of 152 blocks, up to 19 times an attempt, passes 2^31 after 0.74 million attempts).
SG_HD bool sg_reached(unsigned seen, unsigned target) { return (int)(seen - target) >= 0; }
