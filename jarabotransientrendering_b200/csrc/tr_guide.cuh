// tr_guide.cuh - learned directional proposal: MLP (64 -> 3x64 ReLU -> 40) predicting a mixture
// of 8 von Mises-Fisher lobes, trained online on the renderer's own radiance samples.
// No counterpart in the reference renderer.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace trg {

constexpr int kIn = 64;          // padded feature width
constexpr int kHidden = 64;
constexpr int kLobes = 8;
constexpr int kOut = 5 * kLobes; // per lobe: weight logit, mean xyz (unnormalised), concentration
constexpr int kLayers = 4;
constexpr int kParams = kLayers * 64 * 64 + kLayers * 64;   // weights [l][in][out] then biases [l][out]
constexpr int kTile = 128;       // rows per tcgen05 tile (MMA M)
// default number of mbarrier polls before a wait for a CTA's own tensor-core work times out
constexpr uint32_t kWaitPolls = 1u << 24;
// concentration kappa = kKappaMin + kKappaMax * sigmoid(raw - kKappaShift): about exp(raw - 0.4)
// for small kappa (scale-free Adam steps), smoothly saturating at kKappaMax
constexpr float kKappaMin = 0.05f, kKappaMax = 2000.0f, kKappaShift = 8.0f;

// Features of a surface vertex (46 used of 64, rest zero):
//   [0,36)  sin/cos(2^k pi p_d), k = 0..5, d = x,y,z      (p normalised to the scene box)
//   [36,39) p normalised, [39,42) geometric normal, [42,45) outgoing direction (towards the
//   previous vertex), [45] path length / film time length
constexpr int kFeatUsed = 46;

struct GuideDev {
    const uint4* w_fwd;    // 4 canonical K-major B tiles (Wt: [out][in]) bf16, 8 KB each
    const uint4* w_bwd;    // 4 canonical K-major B tiles (W: [in][out]) bf16
    const float* bias;     // [4][64]
    uint32_t spin;         // polls of an mbarrier before a tensor-core wait counts as timed out
};

cudaError_t mlp_forward(const GuideDev& g, const uint4* x, uint32_t m, float* out, int* err, cudaStream_t s);
int mlp_grid(int device);
// CTAs of `kernel` that fit on the device at once (SMs x CTAs per SM, from the kernel's
// registers, shared memory and `tmem_cols` tensor-memory columns per CTA), for persistent loops
int resident_grid(int device, const void* kernel, int threads, size_t dyn_smem, int tmem_cols = 64);
cudaError_t pack_weights(const float* params, uint8_t* w_fwd, uint8_t* w_bwd, cudaStream_t s);
// weight-gradient operands of the four layers
struct DwLayers {
    const uint4* prev[4];      // [m][64] bf16 layer inputs (features, H1, H2, H3)
    const uint4* grad_bf[4];   // [m][64] bf16 gradients w.r.t. the layer outputs
    float* part;               // [layer][CTA][65][64] sums over each CTA's rows: weights, bias
};
struct UpdateArgs {
    const float *part, *loss_part;
    uint32_t nparts, ntiles;
    const int* err;
    int* steps;
    float *loss, *params, *grads, *m1, *m2;
    uint8_t *w_fwd, *w_bwd;
    float lr, c1, c2;
};
// One training step (weight sum, forward + loss gradient + backward, weight gradients, update):
// gradients to grads, the batch loss to *loss, with lr > 0 Adam step `step` and repacked weights.  The
// same bits on every run.  scratch: train_scratch_floats(m); act, dh [3][m][64], dy [m][64] bf16.
struct TrainArgs {
    GuideDev net;
    const uint4* x;
    const float *dirs, *w;
    uint4 *act, *dy, *dh;
    float *scratch, *loss, *params, *grads, *m1, *m2;
    uint8_t *w_fwd, *w_bwd;
    int *err, *steps;          // set when a wait times out; counts the steps applied
    float lr;
    uint32_t step;
};
size_t train_scratch_floats(uint32_t m);
cudaError_t train_step(const TrainArgs& a, uint32_t m, cudaStream_t s);

}  // namespace trg
