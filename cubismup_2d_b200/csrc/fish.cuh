// Fish obstacle support shared by obstacles.cu and fish.cu.
#pragma once
#include "internal.cuh"

namespace cup2d {

struct Ctx;

cudaError_t fish_setup_kernels();          // dynamic shared-memory limits
cudaError_t fish_width_cubes(const FishArrays& F, cudaStream_t st);   // F.w3 from F.width
bool fish_fits_on_chip(int Nm, int nseg, int device);   // staged arrays within the opt-in limit
void launch_fish_midline(Ctx& c, int k, cudaStream_t stream, int mode);
void launch_fish_place(Ctx& c, int k);
void launch_fish_raster(Ctx& c, int k);

// AreaSegment::isIntersectingWithAABB (FishLibrary.cpp:344-401) against the
// block whose first/last cell centres are (start, end).
__device__ __forceinline__ bool segment_hits_block(const Segment& S, const double start[2],
                                                   const double end[2], const double safe)
{
  const double AABB_w[2] = {(end[0] - start[0]) / 2 + safe, (end[1] - start[1]) / 2 + safe};
  const double AABB_c[2] = {(end[0] + start[0]) / 2, (end[1] + start[1]) / 2};
  const double AABB_box[2][2] = {{AABB_c[0] - AABB_w[0], AABB_c[0] + AABB_w[0]},
                                 {AABB_c[1] - AABB_w[1], AABB_c[1] + AABB_w[1]}};
  const double il00 = fmax(S.boxLab[0][0], AABB_box[0][0]), il01 = fmin(S.boxLab[0][1], AABB_box[0][1]);
  const double il10 = fmax(S.boxLab[1][0], AABB_box[1][0]), il11 = fmin(S.boxLab[1][1], AABB_box[1][1]);
  if (il01 - il00 < 0 || il11 - il10 < 0) return false;
  const double widthXbox[2] = {AABB_w[0] * S.normalI[0], AABB_w[0] * S.normalJ[0]};
  const double widthYbox[2] = {AABB_w[1] * S.normalI[1], AABB_w[1] * S.normalJ[1]};
  const double boxBox[2][2] = {
      {AABB_c[0] - widthXbox[0] - widthYbox[0], AABB_c[0] + widthXbox[0] + widthYbox[0]},
      {AABB_c[1] - widthXbox[1] - widthYbox[1], AABB_c[1] + widthXbox[1] + widthYbox[1]}};
  const double if00 = fmax(boxBox[0][0], S.boxObj[0][0]), if01 = fmin(boxBox[0][1], S.boxObj[0][1]);
  const double if10 = fmax(boxBox[1][0], S.boxObj[1][0]), if11 = fmin(boxBox[1][1], S.boxObj[1][1]);
  if (if01 - if00 < 0 || if11 - if10 < 0) return false;
  return true;
}

// a rectangle of blocks clipped to the grid
__device__ __forceinline__ void clip_rect(const GridDesc& g, int& bx0, int& bx1, int& by0, int& by1) {
  bx0 = bx0 < 0 ? 0 : bx0; by0 = by0 < 0 ? 0 : by0;
  bx1 = bx1 > g.bpdx - 1 ? g.bpdx - 1 : bx1; by1 = by1 > g.bpdy - 1 ? g.bpdy - 1 : by1;
}

// Block index range whose cells' AABB, widened by `safe`, can overlap
// [lo, hi] along one axis (one block of margin on each side).
__device__ __forceinline__ void block_range(double lo, double hi, double h, double safe, int& b0, int& b1) {
  if (!(lo <= hi)) { b0 = 1; b1 = 0; return; }            // empty (also for NaN)
  const double bw = BS * h;
  b0 = (int)floor(fmax((lo - safe) / bw, -2.0)) - 1;
  b1 = (int)floor(fmin((hi + safe) / bw, 1e8)) + 1;
}

} // namespace cup2d
