// Tiling of the mesh for the flux kernel.
//
// Cells are stored in Hilbert order of their barycentres, and consecutive
// runs of at most `tile_cells` cells form compact tiles.  One CTA owns one
// tile: it evaluates every face that touches its cells into shared memory
// and sums the fluxes of each cell.  Faces on tile borders are evaluated by
// both adjacent tiles (identical arithmetic, so identical results).
#pragma once

#include <stdint.h>

#include <vector>

#include "ccfd_b200.h"

struct TileSet {
    int n_tiles = 0;
    int tile_cells = 0;
    // faces are numbered tile by tile, each by the first tile that touches
    // it: tile t's own faces are [own_off[t], own_off[t + 1])
    std::vector<int> own_off;    // [n_tiles + 1]
    std::vector<int> face_of;    // [F] reference face of a tile-order face
    std::vector<int> id_of;      // [F] and back
    std::vector<int> border_off; // [n_tiles + 1] offsets into border
    std::vector<int> border;     // tile-order ids of a tile's faces that an earlier tile owns
    std::vector<uint16_t> u_code;  // [4 N] per device cell and side: 2 * local face (own faces, then border) +
                                   // (cell is the neighbour ? 1 : 0), 0xffff padded
    int max_f = 0;
};

// device order of cells (device index -> reference cell): Hilbert curve of
// the barycentres
void ccfd_hilbert_order(const ccfd_mesh* m, std::vector<int>& cell_order);

// device order of cells by reverse Cuthill-McKee on the face-neighbour graph
void ccfd_rcm_order(const ccfd_mesh* m, std::vector<int>& cell_order);

// Build the tiles for a mesh whose cells are already in device order
// (cperm: device -> reference cell, cinv: back).
void ccfd_build_tiles(const ccfd_mesh* m, const std::vector<int>& cperm, const std::vector<int>& cinv, int tile_cells,
                      TileSet& ts);
