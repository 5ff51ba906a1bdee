// tws_grids.h -- making grids for the serving loop.
//
// A grid whose steps run in a batch (or by the plain kernel) needs no share in the
// mesh kernel's workspace, which lies outside a memory budget: create_grid is
// tws_create, without it where `mesh` is false, and a grid that is handed on takes it
// then.
#pragma once

#include "../../include/tws.h"

namespace tws {

int create_grid(int width, int height, const tws_sim_params* params, int flux_storage,
                void* stream, bool mesh, tws_grid** out);
void take_mesh_workspace(tws_grid* g);

}  // namespace tws
