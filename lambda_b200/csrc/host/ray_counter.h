// Indices that traversal lanes take from a counter over n items.
//
// A lane that finds no item left has still counted one up, so the counter ends past n by
// as many as there are lanes (some 300,000 on a B200) and, for n near 2^31, past the
// range of int. Indices are therefore unsigned, which holds n and all lanes.
#pragma once

#ifdef __CUDACC__
#define LAMBDA_HOST_DEVICE __host__ __device__
#else
#define LAMBDA_HOST_DEVICE
#endif

namespace lambda_host {

// The index of the lane at `rank` of a group whose leader found `counter`.
LAMBDA_HOST_DEVICE inline unsigned taken_index(int counter, int rank) { return unsigned(counter) + unsigned(rank); }

// Whether a taken index is one of the n items.
LAMBDA_HOST_DEVICE inline bool item_left(unsigned index, int n) { return index < unsigned(n); }

}  // namespace lambda_host
