/*
 * k_util.cu -- device-wide exclusive scan, the double-double sin
 * coefficients, and the device side of the synthetic trajectory generator.
 */
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "glint_internal.cuh"
#include "scan.cuh"
#include "tracegen.h"

namespace glint {

size_t scan_tmp_bytes(size_t n) {
    const size_t tiles = (n + kScanTile - 1) / kScanTile + 1;
    return sizeof(ScanHead) + tiles * sizeof(unsigned long long);
}

cudaError_t scan_u32(const uint32_t *in, uint32_t *out, size_t n, void *tmp, cudaStream_t s) {
    const bool vec = (((uintptr_t)in | (uintptr_t)out) & 15) == 0;
    return scan_launch(ScanWords{in, vec}, ScanStore{out, vec}, (uint32_t)n, nullptr, tmp, s);
}

/* ---- double-double Taylor coefficients (-1)^k/(2k+1)!, computed on the host
 * in double-double with the same two-product/two-sum steps ---- */
static inline void h_quick(double a, double b, double &s, double &e) {
    s = a + b;
    e = b - (s - a);
}
static inline void h_div(double ah, double al, double d, double &qh, double &ql) {
    double q1 = ah / d;
    double p = q1 * d;
    double pe = std::fma(q1, d, -p);
    double r = ((ah - p) - pe) + al;
    double q2 = r / d;
    h_quick(q1, q2, qh, ql);
}

void init_sin_coef(SinCoef *c) {
    double fh = 1.0, fl = 0.0;
    c->hi[0] = 1.0;
    c->lo[0] = 0.0;
    for (int k = 1; k <= 20; ++k) {
        h_div(fh, fl, (double)(2 * k), fh, fl);
        h_div(fh, fl, (double)(2 * k + 1), fh, fl);
        c->hi[k] = (k & 1) ? -fh : fh;
        c->lo[k] = (k & 1) ? -fl : fl;
    }
}

} // namespace glint

/* ---- device trajectory generator ---- */
struct glint_gen {
    tg_params *d_params = nullptr;
    tg_object *d_objects = nullptr;
    uint32_t n = 0;
    uint32_t step = 0;    /* index of the next step produced */
};

__global__ void k_gen_step(const tg_params *__restrict__ P, tg_object *__restrict__ objs, uint32_t n, uint32_t step,
                           double *__restrict__ out) {
    const tg_params p = *P;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        tg_object o = objs[i];
        if (step > 0) tg_advance(&p, &o, i, step);
        double lon, lat;
        tg_position(&p, &o, &lon, &lat);
        objs[i] = o;
        reinterpret_cast<double2 *>(out)[i] = make_double2(lon, lat);
    }
}

extern "C" {

glint_status glint_gen_create(const void *params, uint32_t params_size, const void *objects, uint32_t num_objects,
                              uint32_t object_size, uint32_t first_step, glint_gen **out) {
    if (!params || !objects || !out || params_size != sizeof(tg_params) || object_size != sizeof(tg_object))
        return GLINT_ERR_INVALID_ARGUMENT;
    glint_gen *g = new glint_gen();
    g->n = num_objects;
    g->step = first_step;
    if (cudaMalloc(&g->d_params, sizeof(tg_params)) != cudaSuccess ||
        cudaMalloc(&g->d_objects, sizeof(tg_object) * (size_t)(num_objects ? num_objects : 1)) != cudaSuccess) {
        cudaFree(g->d_params);
        delete g;
        return GLINT_ERR_OUT_OF_MEMORY;
    }
    cudaMemcpy(g->d_params, params, sizeof(tg_params), cudaMemcpyHostToDevice);
    cudaMemcpy(g->d_objects, objects, sizeof(tg_object) * (size_t)num_objects, cudaMemcpyHostToDevice);
    *out = g;
    return cudaGetLastError() == cudaSuccess ? GLINT_OK : GLINT_ERR_CUDA;
}

glint_status glint_gen_step(glint_gen *g, double *d_out, void *stream) {
    if (!g || !d_out) return GLINT_ERR_INVALID_ARGUMENT;
    unsigned grid = glint::grid_for(g->n, 256, 152u * 16u);
    k_gen_step<<<grid, 256, 0, (cudaStream_t)stream>>>(g->d_params, g->d_objects, g->n, g->step, d_out);
    g->step++;
    return cudaGetLastError() == cudaSuccess ? GLINT_OK : GLINT_ERR_CUDA;
}

glint_status glint_gen_destroy(glint_gen *g) {
    if (!g) return GLINT_OK;
    cudaFree(g->d_params);
    cudaFree(g->d_objects);
    delete g;
    return GLINT_OK;
}

} /* extern "C" */
