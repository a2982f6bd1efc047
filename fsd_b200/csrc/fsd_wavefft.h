// Wave-space transforms for the grid sizes with a register-factored line
// length (wavefft.cu); other grids take the generic passes of mobility.cu.
#pragma once

#include "fsd_internal.h"

namespace fsd {

// Half-spectrum storage: 11 complex fields (green order) of [Nx][Ny][zp]
// with z in [0, Nz / 2], zp padded to a whole 32-byte sector of float2.
inline int wave_zp(int Nz) { return (Nz / 2 + 1 + 3) & ~3; }
// True when every axis has a specialised transform and Ny = Nz.
bool wave_fft_ok(const GridParams& g);
size_t wave_spec_elems(const GridParams& g);   // float2 elements of the half spectra
size_t wave_table_elems(const GridParams& g);  // float4 elements of the Green table
// Wave vectors and the Green's function's scalar factors per half-spectrum point.
void wave_set_table(fsd_handle* h);
// w.grid (6 packed real pairs) -> M_wave spectrum -> w.grid: y and z passes,
// x pass with the Green's function, inverse y and z passes.
void wave_forward_yz(fsd_handle* h);
void wave_x_green(fsd_handle* h);
void wave_inverse_yz(fsd_handle* h);
// Inverse x pass alone, of spectra written to w.spec.
void wave_inverse_x(fsd_handle* h);

}  // namespace fsd
