// fold_route_check.cpp -- which C entry the drop-in's Fold_GPU::calculate_intensity
// takes for each class: the C ABI is replaced by stubs that count the calls
// (no GPU).
#include <cstdio>
#include <cstring>

#include "msosm_gpu_b200.hpp"

using namespace msosm_b200;

static int by_handle = 0, by_pointer = 0;
static msosm_complex series[64];

extern "C" {
const char *msosm_last_error(void) { return ""; }
msosm_status msosm_prepare_nd(float, float, float, unsigned long *nd) { *nd = 0; return MSOSM_OK; }
msosm_status msosm_dedisp_create(const float *, const float *, const float *, int, unsigned long, int, unsigned long,
                                 unsigned int, msosm_dedisp **out)
{
    *out = reinterpret_cast<msosm_dedisp *>(series);
    return MSOSM_OK;
}
msosm_status msosm_dedisp_destroy(msosm_dedisp *) { return MSOSM_OK; }
msosm_status msosm_dedisp_get_info(const msosm_dedisp *, msosm_dedisp_info *i)
{
    std::memset(i, 0, sizeof *i);
    i->M = 16;
    i->fftpoint = 32;
    i->count = 2;
    i->numDMs = 1;
    return MSOSM_OK;
}
msosm_status msosm_dedisp_get_nd(const msosm_dedisp *, unsigned long *) { return MSOSM_OK; }
msosm_status msosm_dedisp_get_delaycount(const msosm_dedisp *, int *) { return MSOSM_OK; }
msosm_status msosm_dedisp_get_delay_points(const msosm_dedisp *, int, int *) { return MSOSM_OK; }
msosm_status msosm_dedisp_get_dedisp_params(const msosm_dedisp *, int, msosm_complex *) { return MSOSM_OK; }
msosm_status msosm_dedisp_output_device_ptr(msosm_dedisp *, msosm_complex **p) { *p = series; return MSOSM_OK; }
msosm_status msosm_fold_create(float, float, unsigned long, unsigned long, msosm_fold **out)
{
    *out = reinterpret_cast<msosm_fold *>(series);
    return MSOSM_OK;
}
msosm_status msosm_fold_get_shape(const msosm_fold *, unsigned long *ps, unsigned long *tb)
{
    *ps = *tb = 4;
    return MSOSM_OK;
}
msosm_status msosm_fold_destroy(msosm_fold *) { return MSOSM_OK; }
msosm_status msosm_fold_planner_destroy(msosm_fold_planner *) { return MSOSM_OK; }
msosm_status msosm_fold_calculate_intensity(msosm_fold *, const msosm_complex *, const msosm_complex *)
{
    ++by_pointer;
    return MSOSM_OK;
}
msosm_status msosm_fold_calculate_intensity_dedisp(msosm_fold *, msosm_dedisp *, msosm_dedisp *)
{
    ++by_handle;
    return MSOSM_OK;
}
}

struct Other {
    msosm_complex *output_buffer_d = series;
};

static bool took(const char *what, int handle, int pointer)
{
    const bool ok = by_handle == handle && by_pointer == pointer;
    if (!ok)
        std::printf("%s: %d by handle, %d by pointer\n", what, by_handle, by_pointer);
    by_handle = by_pointer = 0;
    return ok;
}

int main()
{
    bool ok = true;
    Fold_GPU fold(4.f, 1.f, 32), part(4.f, 1.f, 8);
    MSOSM_GPU_BATCH a(1e6f, 0.f, 1e9f), b(1e6f, 0.f, 1e9f);
    OSM_GPU_BATCH oa(1e6f, 0.f, 1e9f), ob(1e6f, 0.f, 1e9f);
    a.initialize_uint16(32, 2);
    b.initialize_uint16(32, 2);
    oa.initialize_uint16(32, 2);
    ob.initialize_uint16(32, 2);
    Other x, y;
    fold.calculate_intensity(&a, &b);
    ok &= took("MSOSM_GPU_BATCH", 1, 0);
    fold.calculate_intensity<MSOSM_GPU_BATCH>(&a, &b);
    ok &= took("<MSOSM_GPU_BATCH>", 1, 0);
    fold.calculate_intensity(&oa, &ob);
    ok &= took("OSM_GPU_BATCH", 1, 0);
    fold.calculate_intensity<OSM_GPU_BATCH>(&oa, nullptr);
    ok &= took("<OSM_GPU_BATCH>, one polarisation", 1, 0);
    fold.calculate_intensity(&x, &y);
    ok &= took("another class", 0, 1);
    part.calculate_intensity(&oa, &ob);  // the first samples of a longer series
    ok &= took("OSM_GPU_BATCH, a shorter chunk", 0, 1);
    if (ok)
        std::printf("ok\n");
    return ok ? 0 : 1;
}
