// dtrt_gb300 — camera stage of scenes without ray derivatives (static_rays) for nder = 8.
#define DT_CAMERA_STATIC_UNIT
#include "dt_render.cuh"

namespace dt {
template struct CameraStage<8, 0>;
}
