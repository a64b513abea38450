// dtrt_gb300 — questions about a scene description that need no device.
#pragma once
#include <algorithm>

#include "../../include/dtrt_gb300.h"

namespace dt {

// Whether a shape moves: an array of velocities that are all zero (a SceneManager writes one for
// every shape) moves nothing. The array is read only where the vertex count is one that
// scene creation accepts.
inline bool shape_moves(const dtrt_shape_desc &s, int nder) {
    if (!s.velocities || s.num_vertices <= 0) return false;
    const size_t n = (size_t)s.num_vertices * 3 * (nder + (s.normals ? 1 : 0));
    return std::any_of(s.velocities, s.velocities + n, [](float x) { return x != 0.f; });
}

}  // namespace dt
