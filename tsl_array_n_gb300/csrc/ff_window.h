// The choice of the P2G window (k_flip_scatter): the cells around the middle of a
// run of particles whose faces one block sums in shared memory.  Plain C++, so that
// the host can check it for grids no device holds.
#pragma once
#ifdef __CUDACC__
#define FF_WINDOW_FN __host__ __device__ inline
#else
#define FF_WINDOW_FN inline
#endif

constexpr int P2G_CAP = 3096;   // window faces per component: what three blocks an SM leave each

// q20, q80: the 20% and 80% quantiles of the run's cells per axis, n: the grid's cells,
// count: the run's particles.  First cell and extent per axis: the quantiles widened to
// the whole range of an even spread, and the longest axes cut around their middle until
// the window's faces (from one below the first cell to one above the last) fit P2G_CAP.
// Where the run is spread so far that its eight additions a particle and component do
// not reach every face once on average, a window would gather nothing: none (extents 0),
// as for lists in random order and for runs that cross from one plane to the next.
// The product takes 64 bits: a grid one cell thick has less than 2^31 faces, but its
// window before the cut, two faces longer on each axis, can have more.
FF_WINDOW_FN void p2g_window(const int (&q20)[3], const int (&q80)[3], const int (&n)[3], int count, int (&lo)[3],
                             int (&w)[3]) {
    for (int b = 0; b < 3; ++b) {
        const int ext = (q80[b] - q20[b] + 2) / 3;
        const int first = q20[b] - ext, last = q80[b] + ext;
        lo[b] = first > 0 ? first : 0;
        w[b] = (last < n[b] - 1 ? last : n[b] - 1) - lo[b] + 1;
    }
    auto faces = [&] { return (long long)(w[0] + 2) * (w[1] + 2) * (w[2] + 2); };
    if (faces() > 8LL * count) {
        w[0] = w[1] = w[2] = 0;
        return;
    }
    while (faces() > P2G_CAP) {
        const int b = w[0] >= w[1] ? (w[0] >= w[2] ? 0 : 2) : (w[1] >= w[2] ? 1 : 2);
        for (int q = 0; q < 3; ++q)
            if (q == b) {
                const int cut = w[q] / 16 > 1 ? w[q] / 16 : 1;
                lo[q] += cut / 2;
                w[q] -= cut;
            }
    }
}
