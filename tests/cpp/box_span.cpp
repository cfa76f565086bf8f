// box_span of a mesh given by its arrays, for test_box_span.py.
#include "pg_internal.h"

extern "C" int64_t box_span_of(const double *coords, int64_t nv, const int64_t *cells, int64_t nc, const int64_t *bf,
                               const int32_t *tags, int64_t nb) {
    pg_mesh_desc d{};
    d.n_vertices = nv; d.coords = coords;
    d.n_cells = nc; d.cells = cells;
    d.n_boundary_facets = nb; d.bfacet_vertices = bf; d.bfacet_tags = tags;
    pg::HostMesh h;
    return pg::build_mesh(&d, 1.0, h) == 0 ? pg::box_span(h) : -1;
}
