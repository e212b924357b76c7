// The rows of the bands of k_gs_sweep's tiles. Plain C++, so that the rows a
// band stores can be counted without a GPU.
#pragma once

#ifdef __CUDACC__
#define VVM_HOST_DEVICE __host__ __device__
#else
#define VVM_HOST_DEVICE
#endif

namespace vvm {

// Band b of a grid of nz rows (interior 1 .. nz-2) stores the rows k0 .. kl it
// owns; its recurrence starts at ks, up to hz rows below k0. The ghost rows 0
// and nz-1 belong to the bands that own the rows beside them: ks is 1 for every
// band within hz rows of the ground, but only the first may write row 0.
struct GSBand {
    int k0, kl, ks;
    bool bottom, top;   // stores the ghost row 0, nz-1
};
VVM_HOST_DEVICE inline GSBand gs_band(int b, int tr, int hz, int nz) {
    GSBand r;
    r.k0 = 1 + b * tr;
    r.kl = r.k0 + tr - 1 < nz - 2 ? r.k0 + tr - 1 : nz - 2;
    r.ks = r.k0 - hz > 1 ? r.k0 - hz : 1;
    r.bottom = b == 0;
    r.top = r.kl == nz - 2;
    return r;
}

}  // namespace vvm
