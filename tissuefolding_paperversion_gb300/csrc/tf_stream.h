// Whether the FP64 products read their matrix past L2.
#pragma once

#include <cstdint>

namespace tf {

// The products of whole rows read their matrix once an iteration.  Where an iteration
// reads more than L2 holds, the matrix is streamed (evicted first) and L2 keeps the
// vectors and the coarse levels; where it fits, a streamed matrix is read from HBM
// each time all the same.  With the multigrid an iteration reads about twice the
// matrix (its FP16 copy, Q twice, the vectors).  The line, two thirds of L2 (129 MB;
// blocks copied between the two dies' halves take the rest), in us an iteration kept
// / streamed, order-fixed: block-Jacobi CG 18,605 nodes (26 MB) 32.3 / 41.5, 36,980
// 32.9 / 47.8, 61,605 (85 MB) 52.0 / 52.9, 92,480 65.3 / 63.7, 202,005 113.2 / 111.2;
// multigrid 21,125 nodes (29 MB) 99.6 / 109.8 (BiCGStab 182 / 211), 28,880 (40 MB)
// 111 / 122 (225 / 241), 36,980 (51 MB) 144 / 131 (291 / 266), 61,605 179 / 171 (363 /
// 353), 114,005 261 / 258 (534 / 534).  The FP16 sweep's operator is never streamed
// (32 tissues 26.9 -> 27.6 ms a step with it, 320,000 prisms 19.75 -> 19.8).
inline bool stream_matrix(int64_t bytes, bool multigrid, int64_t l2) { return 3 * (multigrid ? 2 : 1) * bytes > 2 * l2; }

}  // namespace tf
