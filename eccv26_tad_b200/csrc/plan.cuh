// Layout of a table's work plan (svtad_plan_build) for the kernels that read it.
#pragma once
#include "common.cuh"

namespace svtad {

constexpr int PLAN_TILE = 128;              // rows of a tile
constexpr int64_t PLAN_MAX_ROWS = 131072;   // one byte of shared memory per row and eighth of the table

struct PlanView {
    const int32_t* order;      // [tiles * PLAN_TILE] rows grouped by which neighbors they have, -1 behind the last
    const uint64_t* mask;      // [tiles] taps that some row of the tile may have
    const int32_t* seq;        // [tiles] tiles, those with most taps first
    const int32_t* count;      // [kk] pairs per tap
    const int32_t* pair_i;     // [kk][n] rows that have the tap, ascending ...
    const int32_t* pair_j;     // [kk][n] ... and the rows their entries name (offsets folded in)
};

inline size_t plan_layout(int64_t n, int kk, const void* base, PlanView* v) {
    const size_t tiles = (size_t)((n + PLAN_TILE - 1) / PLAN_TILE);
    const char* p = static_cast<const char*>(base);
    size_t at = 0;
    auto take = [&](size_t bytes) { const char* q = p + at; at += align_up(bytes, 256); return q; };
    const char* order = take(tiles * PLAN_TILE * 4);
    const char* mask = take(tiles * 8);
    const char* seq = take(tiles * 4);
    const char* count = take((size_t)kk * 4);
    const char* pi = take((size_t)kk * n * 4);
    const char* pj = take((size_t)kk * n * 4);
    if (v != nullptr)
        *v = PlanView{reinterpret_cast<const int32_t*>(order), reinterpret_cast<const uint64_t*>(mask),
                      reinterpret_cast<const int32_t*>(seq), reinterpret_cast<const int32_t*>(count),
                      reinterpret_cast<const int32_t*>(pi), reinterpret_cast<const int32_t*>(pj)};
    return at;
}

}  // namespace svtad
