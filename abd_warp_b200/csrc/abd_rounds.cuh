// The bound of a step's round loop, without CUDA headers (the host tests use it too).
#pragma once

#if defined(__CUDACC__)
#define ABD_ROUNDS __host__ __device__
#else
#define ABD_ROUNDS
#endif

namespace abd {

// May a step's loop start another round (newton.cu), with `rounds` made?  A round makes the kept
// candidate list and then Newton iterations until one leaves the list's region; the round after it
// completes that iteration first, so the iteration that ends round k is the k-th at least, and
// a step of max_iter iterations (one at least) has no round past max_iter + 1.  A step that
// would take one is finished by the host's loop.
ABD_ROUNDS inline bool another_round(int rounds, int max_iter) { return rounds <= (max_iter > 1 ? max_iter : 1); }

}  // namespace abd
