// Host-side helpers shared by the map builder and the API.
#pragma once

#include <stdint.h>

#include "tsdfl.h"

namespace tsdfl {

void set_error(const char* fmt, ...);

uint64_t f2u_x86_host(float v);
float likelihood_value(int mm, float sigma);
float likelihood_init(float sigma);
void code_values(float sigma, float init_value, float out[604]);
void coef_init(tsdfl_map_coef* c, const float mn[3], const float mx[3], float res, float init);
uint64_t host_slot_index(const tsdfl_map_coef& c, const int32_t* grid_occ, float x, float y, float z);
// Largest trunc(offset) that passes the coarse bound check of getIndex
// (cuda_sub_voxel_map.tcc:54-66) on this axis, -1 if none.
int32_t coarse_mmax(uint64_t dim, float res);
// One past the largest brick index trunc(ox) + trunc(oy) up_dim_x + trunc(oz)
// up_dim_2 of offsets that pass the coarse bound check (coarse_mmax, capped at
// 2^22 m) on every axis, with trunc(oz) below `layers`.
uint64_t brick_reach(const tsdfl_map_coef& c, uint64_t layers = UINT64_MAX);
// Bounds below which an offset settles a miss whatever the other axes hold, as
// long as every offset lies below far[0] in magnitude: far[1] on x (an odd
// multiple of 2^63 in the slot index, where sub_dim is even), far[2] on y with
// oz < 1 and far[3] on z (a negative brick index, where no brick row or layer
// reaches past its own end); -1 each, or -inf where the map's shape leaves it
// open.  far[0] is 0 (nothing settled) for resolutions above 1 m.
void miss_bounds(const tsdfl_map_coef& c, int32_t mmax_x, int32_t mmax_y, float far[4]);
// Multipliers of the division-free sub-voxel index q = trunc(fl(s / res)) for
// every float s in [0, 1): returns 2 with *hi such that q == floor(s * hi)
// (exact product), else 1 with (*hi, *lo) such that
// q == trunc(fl(fma(s, hi, fl(s * lo)))), else 0 (no fast path).
int sub_index_mult(float res, uint64_t sub_dim, float* hi, float* lo);

}  // namespace tsdfl
