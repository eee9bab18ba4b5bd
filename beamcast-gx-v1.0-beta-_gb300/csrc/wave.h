// Interface of the wave engine (render.cu) for the other translation units.
#pragma once
#include <cstdint>
#include <vector>

#include "context.h"

namespace bcgx {

constexpr int kMaxGradBounces = 64;

// One view of a render: what a caller asks for, before packing.
struct ViewRequest {
  int scene;        // index into the resident scene set
  bc_camera cam;
  bc_settings s;
  int y0, rows;     // rows [y0, y0 + rows) of the frame
  long long pix_off;  // first pixel of those rows in the frame buffers
  bool want_guides;
};

// Vertex records of a render's paths: for every path and bounce, the material whose
// parameter the vertex depends on and the value the adjoint needs (diffuse: radiance
// gathered before the albedo multiplied the throughput; emitter: throughput times MIS
// weight). m < 0: no record.
struct GradRec {
  int32_t* m;   // [bounce * cap + path]
  float4* v;    // [bounce * cap + path]
  int32_t* nb;  // bounces shaded per path
  int cap;      // paths: those of a wave, or of the whole render when L is given
  float4* L;    // final radiance per path of the whole render (null: records of one wave)
};
size_t grad_rec_bytes(size_t paths, int bounces, bool whole);
GradRec grad_rec_carve(void* p, size_t paths, int bounces, bool whole);

// Gradient render (path replay): adjoint image and parameter map.
struct GradArgs {
  const float* dimg;         // 3 per frame pixel: dLoss / dImage
  const int32_t* mat2param;  // material -> parameter index (-1: not a parameter)
  int n_params;
  double* partial;           // [gradient_grid()][3 * n_params], accumulated over waves
};

// Renders the views; each view's mean radiance ends in render_mean(ctx) at its
// pix_off. With `grad`, also accumulates the path replay gradient into grad->partial;
// with `keep`, leaves the vertex records and radiances of every path there (path
// integrator, fixed samples, the wave engine).
bc_status render_views(bc_context* ctx, const std::vector<ViewRequest>& req, size_t frame_px, int64_t* rays,
                       const GradArgs* grad, const GradRec* keep = nullptr);
// The gradient of one view's `n` paths (sample-major over npix pixels) from kept records;
// collect_timing once the stream has drained (bc_last_timing).
cudaError_t gradient_from_records(bc_context* ctx, const GradRec& rec, long long n, int npix, int spp,
                                  const GradArgs& ga);
void collect_timing(bc_context* ctx);
float* render_mean(bc_context* ctx);

// Photon maps (photon.cu). photon_map_for returns the map of resident scene
// `scene` for the seed, PhotonMapping level and bounces of `s`, from the cache
// or built on the context's stream (then *built_rays is its device ray
// counter), with neighbour lists where a render of `paths` paths wants them; maps
// used after photon_clock() returned `pin` are not evicted.
struct PhotonView;
uint64_t photon_clock(bc_context* ctx);
bc_status photon_map_for(bc_context* ctx, int scene, const bc_settings& s, uint64_t pin, long long paths,
                         PhotonView* view, const unsigned long long** built_rays);
int photon_list_entries(const bc_settings& s);  // neighbour-list entries of the map's capacity
int gradient_grid();
int effective_spp(const bc_settings& s);

}  // namespace bcgx
