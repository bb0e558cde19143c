// Row transforms of the oversampled planes (fft.cu, fft_rows.cuh): one pass over
// memory per axis, fused with the transposes between the grid and the image columns.
#pragma once

#include "curig_internal.h"
#include "kernels.cuh"

namespace curig {

// The passes (fft_rows.cuh).
enum FftMode { X_M2D, Y_M2D, Y_D2M, X_D2M };

constexpr int FFT_PARTS = 8;       // translation units of the kernel instances (fft_lengths.inc)

// Longest row of one unit (fft_lengths.inc); up to twice that in two halves.  A
// half reads the whole row, so in FP32, where the library's long rows are
// good, halves pay from FFT_HALVES32 on (both directions, 12 planes: 4800 3.34 ->
// 3.53 ms, 5400 4.50 -> 4.84, 6000 7.71 -> 6.35, 8192 10.62 -> 9.65); in FP64 at
// every length (4500 7.25 -> 6.13 ms, 6000 18.7 -> 12.4, 8192 26.9 -> 19.8).
constexpr int FFT_LONGEST = 4374, FFT_HALVES32 = 5600;
constexpr int FFT_ZMAX = 1024;     // longest third axis with a pass of its own

// The kernels of one length: X, Y and Z passes, FP32 and FP64.
struct FftKernels {
    const void *x[2] = {}, *y[2] = {}, *z[2] = {};
    const void *x2[2] = {}, *y2[2] = {};   // rows twice as long, two CTAs a row (lengths beyond FFT_LONGEST)
};

// A row length with a pass of its own (index < 0: none, the library's rows).
struct FftPlan {
    int index = -1, n = 0;         // entry of the length table, row length
    int sp = 1;                    // 2: the entry is of half the length, two CTAs a row
    int threads[2] = {}, per[2] = {};      // of a CTA in the X and Y passes: threads, units
    size_t smem[2] = {};
    int stages = 0, R[5] = {};
    int tw_len = 0;                // twiddle table entries (16 bytes each)
};

// Length n in the given element size (4 FP32, 8 FP64; 8 for the Z passes).
bool fft_make_plan(int n, int esize, FftPlan &p);

// What the passes need of the geometry.
struct FftGeom {
    int nx, ny, nf1, nf2, nf3;
    int x0, x1, y0, y1;            // window of the grid that the points reach (even bounds)
#ifdef CURIG_BOUNDS_CHECK
    int *dbg;                      // error flags raised by the index checks
#endif
};

// Twiddle tables of both plans (either may be empty), x first, in the plan's precision.
template <typename T> void launch_fft_tables(const FftPlan &px, const FftPlan &py, void *tw, cudaStream_t st);

// X_M2D / X_D2M: src and dst are the grid and T (or T and the grid); Y_M2D /
// Y_D2M: both are T.
template <typename T>
int launch_fft_pass(FftMode mode, const FftPlan &p, const FftGeom &g, const void *tw, const void *src, void *dst,
                    cudaStream_t st);

// Third axis of the generic 3-D NUFFT: src and dst are T and the modes (m2d) or
// the modes and T; tw: the plan's tables in FP64.
template <typename T>
int launch_fft_z(bool m2d, const FftPlan &p, const DevCorr &cc, const void *tw, const void *src, void *dst,
                 cudaStream_t st);

}  // namespace curig
