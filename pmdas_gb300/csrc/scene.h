// scene.h — host-side scene object and the integrand launcher (internal).
#pragma once

#include <stdint.h>
#include <vector>
#include <cuda_runtime.h>
#include "integrand.h"
#include "grid_types.h"

// The culling lists of a scene (shade.cuh).
size_t mdas_cull_words(const MdasScene& sc);  // 0: the scene kind is not culled
cudaError_t mdas_launch_build_cull(const MdasScene& sc, const float* d_prims, unsigned* lists, cudaStream_t s);

// Evaluates samples [offset, offset+count) of an AoS coordinate buffer with `dim`
// floats per sample (dim >= the scene's own dimension; extra coordinates are
// ignored).  With `counts`, the range is the last adaptive pass's new samples.
// `cull` (may be null) is the scene's culling lists.
cudaError_t mdas_launch_evaluate(const MdasScene& sc, const float* d_prims, const unsigned* cull, const float* coords,
                                 float* values, int dim, const MdasCounts* counts, int offset, int count, int grid,
                                 cudaStream_t s);

cudaError_t mdas_launch_leaf_true_errors(const MdasScene& sc, const float* d_prims, const unsigned* cull,
                                         const MdasDeviceGrid& g, const int* leaves, int L, int samples,
                                         unsigned long long seed, float* out, cudaStream_t s);

// sms: SMs of the device.
cudaError_t mdas_launch_reference_image(const MdasScene& sc, const float* d_prims, const unsigned* cull, int width,
                                        int height, int strata, unsigned long long seed, double* out, int sms,
                                        cudaStream_t s);

int mdas_generate_scene(int kind, uint64_t seed, int count, float scaleX, float scaleY, int width, int height,
                        MdasScene* sc, std::vector<float>* prims);

// Batched integrand over every image's initial samples.  Images of one launch
// share the coordinate stride D.
cudaError_t mdas_launch_evaluate_batch(const MdasBatchScene* scenes, int n, int D, int grid, cudaStream_t s);

// A number that no other scene of the process has had (from 1; integrand.cu).
uint64_t mdas_next_scene_id();

struct mdas_scene {
    // Tells scenes apart for what is kept between calls (the render graph of a grid):
    // a new scene often lies at the address of a destroyed one.
    const uint64_t id = mdas_next_scene_id();
    MdasScene desc;
    std::vector<float> prims;  // host copy
    float* d_prims = nullptr;  // device copy
    unsigned* d_cull = nullptr;  // culling lists of the discs (culled kinds only), rebuilt with every upload
};
