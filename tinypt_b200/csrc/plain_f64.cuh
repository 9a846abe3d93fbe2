// Device view of the f64 scene image and the plain kernel's launch: one lane
// per pixel runs the reference's render worker (src/render.rs:129-205) and
// radiance() (src/integrator.rs:53-135) in f64 over the reference's own
// node, triangle, sphere and instance layouts, found through the FP32 forms'
// trees.
#pragma once

#include "device_common.cuh"
#include "../../include/tinypt_cuda.h"

namespace tpt {

struct PlainScene {
    const NodeF64* nodes;
    const TriF64* tris;
    const MeshF64* meshes;
    const InstanceF64* instances;
    int n_instances;
    const SphereF64* spheres;
    int n_spheres;
    const MaterialF64* mats;
    const LightF64* lights;
    const double* light_cdf;
    int n_lights;
    double light_total;
    int env_kind, env_w, env_h, env_black;  // env_black: env_is_black
    const double* env_data;
    const double* env_row_cdf;
    const double* env_col_cdf;
    double env_total;
    // brackets of the two searches by the variate (make_guide; null: none)
    const uint16_t* env_row_guide;
    const uint16_t* env_col_guide;  // env_col_k + 1 per row
    int env_row_k, env_col_k;
    CameraF64 cam;
    // The FP32 forms' trees (WfScene's arrays) and, per triangle in their
    // leaf order, its place in `tris` (x) and its leaf in `nodes` (y).
    const BvhNode2* nodes32;
    const MeshF32* meshes32;
    const SphereF32* spheres32;
    const int2* links;
    int n_tris;
    int top_root;
    int by_loops;              // geometry_out_of_range: every ray takes the reference's loops
    float top_pad;             // widens the top-level boxes: far above the f64 error of a sphere test
};

struct PlainParams {
    int width, height, spp, max_bounces, rr_start;
    int adaptive, adaptive_min_spp;
    double adaptive_threshold;
    uint64_t seed;
    int row_begin, row_step, n_rows;  // film row k is image row row_begin + k * row_step
};

// counters[0] = samples, [1] = closest-hit rays, [2] = shadow rays, [3] =
// pixels handed out; all zero on entry.
cudaError_t launch_plain(const PlainScene& S, const PlainParams& P, double* acc, double* acc_w, double* acc_sq,
                         unsigned long long* counters, int* flags, int sm_count, cudaStream_t stream);

}  // namespace tpt
