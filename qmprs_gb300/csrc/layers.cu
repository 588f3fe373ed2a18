// (b) per-layer bond-2 truncation + Ran completion, on the dense working state.
//
// Restates MPS.generate_bond_D_unitary_layer (reference
// qmprs/primitives/mps.py:849-891) without an MPS: the bond-2 right-canonical
// form of the working state is its right-to-left truncated SVD, computed one
// cut at a time.  Cut c of state b holds the remainder M (2^c x w, w = 2 r,
// r = bond c+1, row-major, complex64).  k_layer_cut (layer_cut.cuh) forms
// the remainder, reduces its Gram matrix (exact fp32 products, compensated
// sums), diagonalises it, applies quimb's rsum2 cutoff with max_bond 2, fixes
// the singular-vector phases and stores the site tensor.  After the last
// cut, k_layer_build normalises site 0 and turns the n site tensors into n
// gates (mps.py:565-847) in closed form.
#include "layer_cut.cuh"

// fidelity_with_zero_state (mps.py:1020-1039) and the early exit of
// Sequential._get_unitary_layers (sequential.py:390): np.isclose(f, 1, atol).
__global__ void k_layer_fidelity(BatchDev bd, int layer, const float2* work, int num_layers,
                                 double atol, double2* layer_fid, int* nlayers, int* active) {
  grid_wait();
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < bd.B; b += gridDim.x * blockDim.x) {
    if (!active[b]) continue;
    const double2 f = cconj(f2d(work[bd.vec_off[b]]));
    layer_fid[(int64_t)b * num_layers + layer] = f;
    nlayers[b] = layer + 1;
    const double d = cabs_(csub(f, cd(1.0, 0.0)));
    if (d <= atol + 1e-5) active[b] = 0;
  }
}

void launch_layer_cut(const BatchDev& bd, int units, int step, int last, const float2* work, float2* buf0, float2* buf1,
                      int* bonds, double2* vsel, double2* site_t, double2* partials, const int* active,
                      cudaStream_t s) {
  qm_note_launch();
  launch_after(k_layer_cut<CutFast>, units, BLOCK_THREADS, 0, s, bd, step, last, work, bonds, vsel, site_t,
               reinterpret_cast<double*>(partials), buf0, buf1, active);
}

void launch_layer_build(const BatchDev& bd, int layer, const float2* rem0, const float2* rem1,
                        const int* bonds, double2* site_t, double2* gates, signed char* arity,
                        const int* active, cudaStream_t s) {
  qm_note_launch();
  launch_after(k_layer_build<CutFast>, bd.B, BUILD_THREADS, 0, s, bd, layer, rem0, rem1, bonds, site_t, gates, arity,
               active);
}

void launch_layer_fidelity(const BatchDev& bd, int layer, const float2* work, int num_layers,
                           double atol, double2* layer_fid, int* nlayers, int* active,
                           cudaStream_t s) {
  int blocks = (bd.B + 127) / 128;
  qm_note_launch();
  launch_after(k_layer_fidelity, blocks, 128, 0, s, bd, layer, work, num_layers, atol, layer_fid, nlayers, active);
}
