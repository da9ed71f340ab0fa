// mg_layout.h -- the shared-memory layout of a multigrid level or tile, and what follows from it
// for the buffers that hold a copy in that layout.  Plain C++ on the host as well, so that the
// sizes can be checked without a GPU.
#pragma once
#ifdef __CUDACC__
#define MG_HD __host__ __device__ __forceinline__
#else
#define MG_HD inline
#endif

// rows of an odd pitch, so that i + j and the flat index agree in parity up to a constant
MG_HD int mg_pitch(int width) { return width | 1; }

// nodes of one colour: every second flat index of rows x pitch, rounded up (both colours' arrays
// have this length: with an odd number of nodes the second one has an element of padding)
MG_HD int mg_plane(int pitch, int rows) { return (pitch * rows + 1) >> 1; }

// both colours of a whole level of nx x ny cells, ghosts included: the length of its array in
// shared memory and of the copy that a stage starts again from
MG_HD long long mg_level_len(int nx, int ny) { return 2ll * mg_plane(mg_pitch(nx + 3), ny + 3); }
