// qew_poly.cuh -- the FP64 cell-polynomial store.
//
// On a line with one point per field column (n == nx, physical size == Lx)
// every edge midpoint but the wrap edge sits at grid x = e + 1/2, where the
// x weights of the cubic B-spline are the constants w(1/2) = 1/48, 23/48,
// 23/48, 1/48 (filtered_noise.h:33-44 at t = 1/2). Along y, inside row cell
// j the interpolant is a cubic in the fraction t (filtered_noise.h:33-62) of
// the x-filtered coefficients E_b of rows j-1 .. j+2. The store keeps, per
// (row cell j, column e), that cubic as four 64-bit fixed-point numbers
// (FxCubic, qew_fix.cuh) in a unit of the cell's own, taken once when the field
// is built from the same integers that the 16-tap gather forms at each call:
// where dx and dy are powers of two, an edge's dV/dy and V are the same bits with
// the store and without. (The linear gradient's walk adds heights and both edges
// in integers before it rounds, and a dy that is no power of two locates a row
// on the store by one product, so gradients agree to rounding.) A gradient edge
// then reads one aligned 32-byte cell and evaluates two integer products, where
// the reference's order (filtered_noise.h:159-176) reads 16 taps.
#pragma once

#include "qew_internal.cuh"

// Builds the store of a field's FP64 coefficients c ([ny][nx], x fastest)
// into out ([ny][nx][4], 32-byte aligned), on ctx's stream; max_bits: the bit
// pattern of the largest |c|, on the device.
qew_status qew_poly_store_build(qew_ctx *ctx, const double *c, int nx, int ny,
                                const unsigned long long *max_bits, long long *out);
// FP64 gradient of `count` lines (n apart) on the store; QEW_ERR_UNSUPPORTED
// (no error recorded) when the field holds no store or the line does not
// have one point per field column.
qew_status qew_gradient_poly_enqueue(qew_ctx *ctx, const qew_field *f, int count,
                                     const double *d_h, int n, const qew_params *p,
                                     double *d_grad,
                                     bool host_grad = false);
