// Explicit instantiation of the C=1 kernels (one translation unit per spinor
// size so that the build compiles them in parallel).
#include <vector>

#include "gpe_kernels.cuh"
#include "gpe_observe.cuh"

namespace gpe {
GPE_INSTANTIATE(float, 1)
GPE_INSTANTIATE_OBSERVE(float, 1)
GPE_INSTANTIATE_OBSERVE(double, 1)
GPE_INSTANTIATE(double, 1)
GPE_INSTANTIATE_TILE(float, 1)
GPE_INSTANTIATE_TILE(double, 1)
GPE_INSTANTIATE_MARCH(float, 1)
GPE_INSTANTIATE_MARCH(double, 1)
GPE_INSTANTIATE_SLAB(float, 1)
GPE_INSTANTIATE_SLAB(double, 1)
GPE_INSTANTIATE_ROWS(float, 1)
GPE_INSTANTIATE_ROWS(double, 1)
GPE_INSTANTIATE_INIT(float, 1)
GPE_INSTANTIATE_INIT(double, 1)
GPE_INSTANTIATE_HYPER_TILE(float, 1)
GPE_INSTANTIATE_HYPER_TILE(double, 1)
template cudaError_t launch_split<float>(const StepArgs&, int, double, cudaStream_t);
template cudaError_t launch_split<double>(const StepArgs&, int, double, cudaStream_t);

cudaError_t launch_dot(const StepArgs& a, int precision, int C, cudaStream_t s) {
    if (precision == GPE_FP64) {
        if (C == 1) return launch_dot_t<double, 1>(a, s);
        if (C == 3) return launch_dot_t<double, 3>(a, s);
        return launch_dot_t<double, 5>(a, s);
    }
    if (C == 1) return launch_dot_t<float, 1>(a, s);
    if (C == 3) return launch_dot_t<float, 3>(a, s);
    return launch_dot_t<float, 5>(a, s);
}

cudaError_t launch_pack_any(int precision, double* packed, char* dev_base, uint32_t X, uint32_t Y, uint32_t Z,
                            uint32_t vals, size_t pitch, size_t slice, bool to_device, cudaStream_t s) {
    if (precision == GPE_FP64) return launch_pack<double>(packed, dev_base, X, Y, Z, vals, pitch, slice, to_device, s);
    return launch_pack<float>(packed, dev_base, X, Y, Z, vals, pitch, slice, to_device, s);
}
GPE_INSTANTIATE_IL(1)

cudaError_t launch_split_planes(const StepArgs& a, int part, char* const planes[4], const Grid& g, const int32_t* tab,
                                cudaStream_t s) {
    // planes: R, I, q_R, q_I
    const SplitPlanes p = {planes[part], planes[1 - part], planes[2 + part], planes[3 - part]};
    return launch_line_split(a, part, p, make_line_grid(g, g.V), make_line_grid(g, g.E), tab, s);
}
cudaError_t launch_split_planes_convert(char* psi, char* q, char* const planes[4], const Grid& g, bool to_planes, cudaStream_t s) {
    const cudaError_t e = launch_split_convert(psi, g.pitch, g.slice, g.cell_bytes, planes[0], planes[1], make_line_grid(g, g.V),
                                               to_planes, false, s);
    if (e != cudaSuccess) return e;
    return launch_split_convert(q, g.qpitch, g.qslice, g.qcell_bytes, planes[2], planes[3], make_line_grid(g, g.E), to_planes, true,
                                s);
}
size_t split_plane_bytes(const Grid& g, bool q) { return make_line_grid(g, q ? g.E : g.V).bytes; }
bool split_planes_fit(const Grid& g) { return line_fits(make_line_grid(g, g.V)) && line_fits(make_line_grid(g, g.E)); }
void split_plane_table(const Grid& g, const gpe_incidence* inc, const gpe_edge* edges, std::vector<int32_t>& tab) {
    const LineGrid G = make_line_grid(g, g.V);
    auto cells = [&](int dx, int dy, int dz) { return (dz * (int32_t)G.Yp + dy) * (int32_t)G.Xp + dx; };
    tab.clear();
    for (uint32_t i = 0; i < 4 * g.V; ++i) {
        tab.push_back(cells(inc[i].dx, inc[i].dy, inc[i].dz));
        tab.push_back((int32_t)inc[i].edge);
    }
    for (uint32_t i = 0; i < g.E; ++i) {
        tab.push_back(cells(edges[i].dx, edges[i].dy, edges[i].dz));
        tab.push_back((int32_t)edges[i].to);
    }
    for (uint32_t i = 0; i < g.E; ++i) tab.push_back((int32_t)edges[i].from);
}
GPE_DEFINE_IL_CONVERT
}  // namespace gpe
