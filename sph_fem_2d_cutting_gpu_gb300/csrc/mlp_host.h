// mlp_host.h -- the host-side MLP object (sph_mlp) shared by the MLP entry
// points and the context's warm-start attachment.
#pragma once

#include <mutex>
#include <string>
#include <vector>

#include "launch.cuh"

struct sph_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    int num_sms = 0;
    float *params = nullptr, *m1 = nullptr, *m2 = nullptr;   // FP32 parameters and Adam moments
    uint16_t *wb = nullptr;                                  // BF16 weight copies
    float *part = nullptr;                                   // per-CTA gradient partials
    int part_rows = 0;
    float *grad = nullptr;                                   // [kMlpParams + 1], then the status word
    float *loss = nullptr;                                   // per-step losses of a training run
    int64_t loss_cap = 0;
    uint32_t *status = nullptr;
    // Scratch kept for the next call: a batch's features and targets on the device (up to
    // kKeepSamples), and a page-locked copy of gradient, loss and status.
    float *batch = nullptr;
    int64_t batch_cap = 0;
    float *result = nullptr;
    // Held by every call that uses the scratch, the stream, the parameters or the norm, a
    // context's attachment included: one at a time.
    mutable std::mutex busy;
    sph_mlp_norm norm{};
    int64_t adam_t = 0;
    std::vector<void *> allocs;
    std::string err;
};

namespace sphfem {
MlpDev mlp_view(const sph_mlp *m, const float *params, const uint16_t *wb);
}
