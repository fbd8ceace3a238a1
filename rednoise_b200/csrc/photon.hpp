// Photon mapping with reference semantics (photon.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "refmode.hpp"

namespace rnb {

constexpr int kMaxPhotons = 1 << 22;

// How many diffuse hits pass 2 keeps at a time (84 bytes of scratch each): two per pixel, or one
// row's 16 per pixel where that is more, up to 2^24 (1.4 GB); with `fewest` up to 2^18 (22 MB),
// for when memory is short. None with a final gather, which works pixel by pixel.
size_t photon_requests(int width, int height, int gather_rays, bool fewest);

// Device scratch the photon mapper needs for n_photons photons and that many requests.
cudaError_t photon_scratch_bytes(int n_photons, size_t requests, size_t &bytes);

// Both passes of renderPhotonMapped into argb (device, width*height 0xAARRGGBB).
// hp: host copy of the parameters (lights[0] emits); d_params: the same on the
// device. requests: of photon_requests. Synchronises st to size the deposit pass (twice where
// the photons take more than ten draws on average) and, without a final gather, once per
// band of rows; deposits_out receives the number of stored photons.
cudaError_t launch_photon_mapped(const SceneView &sv, const float4 *ref_shade, const RefParams &hp,
                                 const RefParams *d_params, int n_photons, int gather_rays, size_t requests,
                                 void *scratch, size_t scratch_bytes, uint32_t *argb, int *status, cudaStream_t st,
                                 unsigned *deposits_out);

} // namespace rnb
