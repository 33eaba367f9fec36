// Host build of Facets (cpabdiffeo_b200/csrc/cpab_cell.cuh) for tests/test_cell_facets_host.py.
#include "cpab_cell.cuh"

using namespace cpab;

// For pairs (p, q): the exact cell of each, and the float margin of q to the facets of p's cell.
template <int DIM, int TESS>
static void margins(const Tess &t, const double *p, const double *q, int *cp, int *cq, float *m, long n)
{
    for (long i = 0; i < n; ++i) {
        cp[i] = exact_cell<DIM, TESS>(t, p + i * DIM);
        cq[i] = exact_cell<DIM, TESS>(t, q + i * DIM);
        Facets<DIM, TESS> f;
        int kb[DIM];
        cell_box<DIM, TESS>(t, cp[i], kb);
        f.enter(t, cp[i], kb);
        float r[DIM];
        for (int k = 0; k < DIM; ++k) r[k] = (float)fma(q[i * DIM + k], t.inv_inc[k], -((double)kb[k] + 0.5));
        m[i] = f.margin(r);
    }
}

extern "C" int facet_margins(int dim, int tess, const int *nCs, const double *incs, const double *p, const double *q,
                             int *cp, int *cq, float *m, long n)
{
    Tess t;
    if (!make_tess(dim, tess, nCs, incs, t)) return 0;
    if (dim == 1) margins<1, 2>(t, p, q, cp, cq, m, n);
    else if (dim == 2) tess == 1 ? margins<2, 1>(t, p, q, cp, cq, m, n) : margins<2, 2>(t, p, q, cp, cq, m, n);
    else tess == 1 ? margins<3, 1>(t, p, q, cp, cq, m, n) : margins<3, 2>(t, p, q, cp, cq, m, n);
    return 1;
}
