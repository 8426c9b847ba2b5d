// s2d_frame.cuh -- index arithmetic of the framed images of the closure's fused
// forward (also compiles as C++).
//
// An image of n x n pixels carries a one-pixel circular frame: framed pixel f
// of a row is image pixel f - 1, the frame pixels 0 and n + 1 are the image's
// last and first.  Rows are net_pitch(n) pixels long, an even number, so an odd
// n has one pixel more that no output reads.
#pragma once

#ifdef __CUDACC__
#define S2D_FRAME_HD __host__ __device__ __forceinline__
#else
#define S2D_FRAME_HD inline
#endif

namespace s2d {

S2D_FRAME_HD int net_pitch(int n) { return (n + 3) & ~1; }

// The image pixel (or row) whose copy stands at framed position f, 0 <= f <
// net_pitch(n); the padding holds the image's pixel 0 as well.
S2D_FRAME_HD int net_frame_source(int f, int n) { return f == 0 ? n - 1 : (f > n ? 0 : f - 1); }

}  // namespace s2d
