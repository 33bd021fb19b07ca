// gnm_tensor.h — split-BF16 tcgen05 engine and the backward kernel (host entry points).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

struct gnm_plan;
struct gnm_prep_view;

namespace gnm {

// AUTO picks the tensor engine from this many score columns on.  Its cost alone
// would put the line lower (20,000 x 200,000: 16 scores take 0.41 ms, one score
// on the plain engine 0.31); it stays where the plain engine's sums, on another
// grid, have always ended, so that a call's result does not move.
constexpr uint64_t kTensorMinScores = 8;

// Smallest row block the end-to-end call splits the tensor engine's rows into.
constexpr uint64_t kTensorMinBlock = 16384;

struct PhaseTrace;
// Builds the limb planes from the caller's CSR (read during the call only).
void tensor_plan_create(gnm_plan* p, const gnm_prep_view* prep, PhaseTrace* trace);
void tensor_plan_destroy(gnm_plan* p);
void tensor_reset(gnm_plan* p, cudaStream_t s);
// Up to 64 scores a shape chooses between people as the MMA's M (the default)
// and the wide kernels (scores as M); over 64 see tensor_default_shape.
bool tensor_can_narrow(const gnm_plan* p);
// Shape codes: raster order of the wide kernels | narrow << 1 | 8-bit limbs << 2 |
// SM pairs << 3 | kShapeExact (gnm_plan_set_shape).  A code with kShapeExact always
// means the kernel that its other bits name; without it, over 64 scores, the
// default shape stands for whichever kernel the plan prefers.
constexpr uint32_t kShapeExact = 16;
uint32_t tensor_shape(const gnm_plan* p);
uint32_t tensor_default_shape(const gnm_plan* p);
// A shape that runs people as M.
uint32_t tensor_people_shape(const gnm_plan* p);
// The code that names the kernel which runs the plan's blocks in a shape.
uint32_t tensor_exact(const gnm_plan* p, uint32_t shape);
void tensor_set_shape(gnm_plan* p, uint32_t shape);
void tensor_accumulate(gnm_plan* p, const uint8_t* d_rows, uint64_t pitch, uint64_t v0,
                       uint64_t nv, cudaStream_t s);
void tensor_finalize(gnm_plan* p, double* d_sums, uint32_t* d_counts, bool add_baseline,
                     cudaStream_t s);
void backward_dw(gnm_plan* p, const uint8_t* d_rows, uint64_t pitch, const float* d_grad_s,
                 float* d_grad_w, float* d_grad_corr, cudaStream_t s);

}  // namespace gnm
