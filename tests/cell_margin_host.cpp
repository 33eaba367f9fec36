// Host build of fast_cell_3d_tet_m and cell_box (cpabdiffeo_b200/csrc/cpab_cell.cuh) for
// tests/test_cell_margin_host.py.
#include "cpab_cell.cuh"

using namespace cpab;

template <int DIM, int TESS>
static int boxes(const Tess &t, int *kb)
{
    for (int c = 0; c < t.nC; ++c) cell_box<DIM, TESS>(t, c, kb + c * DIM);
    return t.nC;
}

extern "C" int cell_boxes(int dim, int tess, const int *nCs, const double *incs, int *kb)
{
    Tess t;
    if (!make_tess(dim, tess, nCs, incs, t)) return 0;
    if (dim == 1) return boxes<1, 2>(t, kb);
    if (dim == 2) return tess == 1 ? boxes<2, 1>(t, kb) : boxes<2, 2>(t, kb);
    return tess == 1 ? boxes<3, 1>(t, kb) : boxes<3, 2>(t, kb);
}

extern "C" int tet_margins(const int *nCs, const double *incs, const float *pts, int *plain, int *with_m, float *m, long n)
{
    Tess t;
    if (!make_tess(3, 1, nCs, incs, t)) return 0;
    for (long i = 0; i < n; ++i) {
        plain[i] = fast_cell<3, 1>(t, pts + i * 3);
        with_m[i] = fast_cell_3d_tet_m(t, pts + i * 3, m[i]);
    }
    return 1;
}
