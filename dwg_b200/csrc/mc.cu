// mc.cu -- marching cubes, two passes with cell-ordered (deterministic) output.
//
// The reference (src/TurboMC.cu:383-478) launches one 12-thread block per cell
// and appends triangles at atomicAdd slots.  Here pass 1 counts the triangles
// of every 256 cells; a scan gives each such block its output offset; pass 2
// visits the blocks that have triangles and writes each at its final
// position, so the triangle order is the cell order (x fastest) -- identical
// from run to run.
//
// Conventions kept from the reference: corner c of cell (x,y,z) sits at
// (x + (b0 != b1), y + b1, z + !b2) (src/TurboMC.cu:408-413); bit c of the case
// index is set when the corner value is above the iso value (:418-425); edge e
// joins corners (e & 7, e<4 ? (e+1)&3 : e<8 ? 4+((e-3)&3) : e-4) (:433-434);
// vertex = P1 - l (P2 - P1), l = (v1 - iso)/(v2 - v1 + 1e-10) (:373-381);
// centroid = mean of the vertices; normal = -cross/(|cross| + 1e-8) (:453-470);
// the triangles of each case are the reference's (kTriangles below), checked
// against the polygons the cube geometry gives (mc_tables_host).
#include <cub/cub.cuh>

#include <algorithm>
#include <mutex>

#include "mc.cuh"

namespace dwg {

__constant__ __align__(16) signed char c_tri[256][16];
__constant__ unsigned char c_ntri[256];
__constant__ unsigned short c_edges[256];
// the same in global memory, for blocks that stage them in shared memory (a
// constant load serves one address at a time)
__device__ __align__(16) signed char g_tri[256][16];
__device__ __align__(16) unsigned char g_ntri[256];

static const int kCorner[8][3] = {{0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1},
                                  {0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}};
static int edge_a(int e) { return e & 7; }
static int edge_b(int e) { return e < 4 ? ((e + 1) & 3) : (e < 8 ? 4 + ((e - 3) & 3) : e - 4); }

// Triangles of each of the 256 cases, as edge-index triples: the reference's
// per-case triangle lists (src/TurboMC.cu:57-314), kept equal on purpose.
// The DWG iteration pushes every triangle's unit normal onto the 15 nearest
// points of its centroid, so splitting a 4-7-gon along other diagonals changes
// the reconstruction, not only the mesh (measured on BASELINE config 1 with
// the FP64 oracle: 0.965 leaf-orientation agreement between the two splits).
static const signed char kTriangles[256][16] = {
    {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 3, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 1, 9, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 8, 3, 9, 8, 1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 10, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 3, 1, 2, 10, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {9, 2, 10, 0, 2, 9, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {2, 8, 3, 2, 10, 8, 10, 9, 8, -1, -1, -1, -1, -1, -1, -1},
    {3, 11, 2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 11, 2, 8, 11, 0, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 9, 0, 2, 3, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 11, 2, 1, 9, 11, 9, 8, 11, -1, -1, -1, -1, -1, -1, -1},
    {3, 10, 1, 11, 10, 3, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 10, 1, 0, 8, 10, 8, 11, 10, -1, -1, -1, -1, -1, -1, -1},
    {3, 9, 0, 3, 11, 9, 11, 10, 9, -1, -1, -1, -1, -1, -1, -1},
    {9, 8, 10, 10, 8, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 7, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 3, 0, 7, 3, 4, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 1, 9, 8, 4, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 1, 9, 4, 7, 1, 7, 3, 1, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 10, 8, 4, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {3, 4, 7, 3, 0, 4, 1, 2, 10, -1, -1, -1, -1, -1, -1, -1},
    {9, 2, 10, 9, 0, 2, 8, 4, 7, -1, -1, -1, -1, -1, -1, -1},
    {2, 10, 9, 2, 9, 7, 2, 7, 3, 7, 9, 4, -1, -1, -1, -1},
    {8, 4, 7, 3, 11, 2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {11, 4, 7, 11, 2, 4, 2, 0, 4, -1, -1, -1, -1, -1, -1, -1},
    {9, 0, 1, 8, 4, 7, 2, 3, 11, -1, -1, -1, -1, -1, -1, -1},
    {4, 7, 11, 9, 4, 11, 9, 11, 2, 9, 2, 1, -1, -1, -1, -1},
    {3, 10, 1, 3, 11, 10, 7, 8, 4, -1, -1, -1, -1, -1, -1, -1},
    {1, 11, 10, 1, 4, 11, 1, 0, 4, 7, 11, 4, -1, -1, -1, -1},
    {4, 7, 8, 9, 0, 11, 9, 11, 10, 11, 0, 3, -1, -1, -1, -1},
    {4, 7, 11, 4, 11, 9, 9, 11, 10, -1, -1, -1, -1, -1, -1, -1},
    {9, 5, 4, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {9, 5, 4, 0, 8, 3, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 5, 4, 1, 5, 0, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {8, 5, 4, 8, 3, 5, 3, 1, 5, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 10, 9, 5, 4, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {3, 0, 8, 1, 2, 10, 4, 9, 5, -1, -1, -1, -1, -1, -1, -1},
    {5, 2, 10, 5, 4, 2, 4, 0, 2, -1, -1, -1, -1, -1, -1, -1},
    {2, 10, 5, 3, 2, 5, 3, 5, 4, 3, 4, 8, -1, -1, -1, -1},
    {9, 5, 4, 2, 3, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 11, 2, 0, 8, 11, 4, 9, 5, -1, -1, -1, -1, -1, -1, -1},
    {0, 5, 4, 0, 1, 5, 2, 3, 11, -1, -1, -1, -1, -1, -1, -1},
    {2, 1, 5, 2, 5, 8, 2, 8, 11, 4, 8, 5, -1, -1, -1, -1},
    {10, 3, 11, 10, 1, 3, 9, 5, 4, -1, -1, -1, -1, -1, -1, -1},
    {4, 9, 5, 0, 8, 1, 8, 10, 1, 8, 11, 10, -1, -1, -1, -1},
    {5, 4, 0, 5, 0, 11, 5, 11, 10, 11, 0, 3, -1, -1, -1, -1},
    {5, 4, 8, 5, 8, 10, 10, 8, 11, -1, -1, -1, -1, -1, -1, -1},
    {9, 7, 8, 5, 7, 9, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {9, 3, 0, 9, 5, 3, 5, 7, 3, -1, -1, -1, -1, -1, -1, -1},
    {0, 7, 8, 0, 1, 7, 1, 5, 7, -1, -1, -1, -1, -1, -1, -1},
    {1, 5, 3, 3, 5, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {9, 7, 8, 9, 5, 7, 10, 1, 2, -1, -1, -1, -1, -1, -1, -1},
    {10, 1, 2, 9, 5, 0, 5, 3, 0, 5, 7, 3, -1, -1, -1, -1},
    {8, 0, 2, 8, 2, 5, 8, 5, 7, 10, 5, 2, -1, -1, -1, -1},
    {2, 10, 5, 2, 5, 3, 3, 5, 7, -1, -1, -1, -1, -1, -1, -1},
    {7, 9, 5, 7, 8, 9, 3, 11, 2, -1, -1, -1, -1, -1, -1, -1},
    {9, 5, 7, 9, 7, 2, 9, 2, 0, 2, 7, 11, -1, -1, -1, -1},
    {2, 3, 11, 0, 1, 8, 1, 7, 8, 1, 5, 7, -1, -1, -1, -1},
    {11, 2, 1, 11, 1, 7, 7, 1, 5, -1, -1, -1, -1, -1, -1, -1},
    {9, 5, 8, 8, 5, 7, 10, 1, 3, 10, 3, 11, -1, -1, -1, -1},
    {5, 7, 0, 5, 0, 9, 7, 11, 0, 1, 0, 10, 11, 10, 0, -1},
    {11, 10, 0, 11, 0, 3, 10, 5, 0, 8, 0, 7, 5, 7, 0, -1},
    {11, 10, 5, 7, 11, 5, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {10, 6, 5, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 3, 5, 10, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {9, 0, 1, 5, 10, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 8, 3, 1, 9, 8, 5, 10, 6, -1, -1, -1, -1, -1, -1, -1},
    {1, 6, 5, 2, 6, 1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 6, 5, 1, 2, 6, 3, 0, 8, -1, -1, -1, -1, -1, -1, -1},
    {9, 6, 5, 9, 0, 6, 0, 2, 6, -1, -1, -1, -1, -1, -1, -1},
    {5, 9, 8, 5, 8, 2, 5, 2, 6, 3, 2, 8, -1, -1, -1, -1},
    {2, 3, 11, 10, 6, 5, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {11, 0, 8, 11, 2, 0, 10, 6, 5, -1, -1, -1, -1, -1, -1, -1},
    {0, 1, 9, 2, 3, 11, 5, 10, 6, -1, -1, -1, -1, -1, -1, -1},
    {5, 10, 6, 1, 9, 2, 9, 11, 2, 9, 8, 11, -1, -1, -1, -1},
    {6, 3, 11, 6, 5, 3, 5, 1, 3, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 11, 0, 11, 5, 0, 5, 1, 5, 11, 6, -1, -1, -1, -1},
    {3, 11, 6, 0, 3, 6, 0, 6, 5, 0, 5, 9, -1, -1, -1, -1},
    {6, 5, 9, 6, 9, 11, 11, 9, 8, -1, -1, -1, -1, -1, -1, -1},
    {5, 10, 6, 4, 7, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 3, 0, 4, 7, 3, 6, 5, 10, -1, -1, -1, -1, -1, -1, -1},
    {1, 9, 0, 5, 10, 6, 8, 4, 7, -1, -1, -1, -1, -1, -1, -1},
    {10, 6, 5, 1, 9, 7, 1, 7, 3, 7, 9, 4, -1, -1, -1, -1},
    {6, 1, 2, 6, 5, 1, 4, 7, 8, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 5, 5, 2, 6, 3, 0, 4, 3, 4, 7, -1, -1, -1, -1},
    {8, 4, 7, 9, 0, 5, 0, 6, 5, 0, 2, 6, -1, -1, -1, -1},
    {7, 3, 9, 7, 9, 4, 3, 2, 9, 5, 9, 6, 2, 6, 9, -1},
    {3, 11, 2, 7, 8, 4, 10, 6, 5, -1, -1, -1, -1, -1, -1, -1},
    {5, 10, 6, 4, 7, 2, 4, 2, 0, 2, 7, 11, -1, -1, -1, -1},
    {0, 1, 9, 4, 7, 8, 2, 3, 11, 5, 10, 6, -1, -1, -1, -1},
    {9, 2, 1, 9, 11, 2, 9, 4, 11, 7, 11, 4, 5, 10, 6, -1},
    {8, 4, 7, 3, 11, 5, 3, 5, 1, 5, 11, 6, -1, -1, -1, -1},
    {5, 1, 11, 5, 11, 6, 1, 0, 11, 7, 11, 4, 0, 4, 11, -1},
    {0, 5, 9, 0, 6, 5, 0, 3, 6, 11, 6, 3, 8, 4, 7, -1},
    {6, 5, 9, 6, 9, 11, 4, 7, 9, 7, 11, 9, -1, -1, -1, -1},
    {10, 4, 9, 6, 4, 10, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 10, 6, 4, 9, 10, 0, 8, 3, -1, -1, -1, -1, -1, -1, -1},
    {10, 0, 1, 10, 6, 0, 6, 4, 0, -1, -1, -1, -1, -1, -1, -1},
    {8, 3, 1, 8, 1, 6, 8, 6, 4, 6, 1, 10, -1, -1, -1, -1},
    {1, 4, 9, 1, 2, 4, 2, 6, 4, -1, -1, -1, -1, -1, -1, -1},
    {3, 0, 8, 1, 2, 9, 2, 4, 9, 2, 6, 4, -1, -1, -1, -1},
    {0, 2, 4, 4, 2, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {8, 3, 2, 8, 2, 4, 4, 2, 6, -1, -1, -1, -1, -1, -1, -1},
    {10, 4, 9, 10, 6, 4, 11, 2, 3, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 2, 2, 8, 11, 4, 9, 10, 4, 10, 6, -1, -1, -1, -1},
    {3, 11, 2, 0, 1, 6, 0, 6, 4, 6, 1, 10, -1, -1, -1, -1},
    {6, 4, 1, 6, 1, 10, 4, 8, 1, 2, 1, 11, 8, 11, 1, -1},
    {9, 6, 4, 9, 3, 6, 9, 1, 3, 11, 6, 3, -1, -1, -1, -1},
    {8, 11, 1, 8, 1, 0, 11, 6, 1, 9, 1, 4, 6, 4, 1, -1},
    {3, 11, 6, 3, 6, 0, 0, 6, 4, -1, -1, -1, -1, -1, -1, -1},
    {6, 4, 8, 11, 6, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {7, 10, 6, 7, 8, 10, 8, 9, 10, -1, -1, -1, -1, -1, -1, -1},
    {0, 7, 3, 0, 10, 7, 0, 9, 10, 6, 7, 10, -1, -1, -1, -1},
    {10, 6, 7, 1, 10, 7, 1, 7, 8, 1, 8, 0, -1, -1, -1, -1},
    {10, 6, 7, 10, 7, 1, 1, 7, 3, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 6, 1, 6, 8, 1, 8, 9, 8, 6, 7, -1, -1, -1, -1},
    {2, 6, 9, 2, 9, 1, 6, 7, 9, 0, 9, 3, 7, 3, 9, -1},
    {7, 8, 0, 7, 0, 6, 6, 0, 2, -1, -1, -1, -1, -1, -1, -1},
    {7, 3, 2, 6, 7, 2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {2, 3, 11, 10, 6, 8, 10, 8, 9, 8, 6, 7, -1, -1, -1, -1},
    {2, 0, 7, 2, 7, 11, 0, 9, 7, 6, 7, 10, 9, 10, 7, -1},
    {1, 8, 0, 1, 7, 8, 1, 10, 7, 6, 7, 10, 2, 3, 11, -1},
    {11, 2, 1, 11, 1, 7, 10, 6, 1, 6, 7, 1, -1, -1, -1, -1},
    {8, 9, 6, 8, 6, 7, 9, 1, 6, 11, 6, 3, 1, 3, 6, -1},
    {0, 9, 1, 11, 6, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {7, 8, 0, 7, 0, 6, 3, 11, 0, 11, 6, 0, -1, -1, -1, -1},
    {7, 11, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {7, 6, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {3, 0, 8, 11, 7, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 1, 9, 11, 7, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {8, 1, 9, 8, 3, 1, 11, 7, 6, -1, -1, -1, -1, -1, -1, -1},
    {10, 1, 2, 6, 11, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 10, 3, 0, 8, 6, 11, 7, -1, -1, -1, -1, -1, -1, -1},
    {2, 9, 0, 2, 10, 9, 6, 11, 7, -1, -1, -1, -1, -1, -1, -1},
    {6, 11, 7, 2, 10, 3, 10, 8, 3, 10, 9, 8, -1, -1, -1, -1},
    {7, 2, 3, 6, 2, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {7, 0, 8, 7, 6, 0, 6, 2, 0, -1, -1, -1, -1, -1, -1, -1},
    {2, 7, 6, 2, 3, 7, 0, 1, 9, -1, -1, -1, -1, -1, -1, -1},
    {1, 6, 2, 1, 8, 6, 1, 9, 8, 8, 7, 6, -1, -1, -1, -1},
    {10, 7, 6, 10, 1, 7, 1, 3, 7, -1, -1, -1, -1, -1, -1, -1},
    {10, 7, 6, 1, 7, 10, 1, 8, 7, 1, 0, 8, -1, -1, -1, -1},
    {0, 3, 7, 0, 7, 10, 0, 10, 9, 6, 10, 7, -1, -1, -1, -1},
    {7, 6, 10, 7, 10, 8, 8, 10, 9, -1, -1, -1, -1, -1, -1, -1},
    {6, 8, 4, 11, 8, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {3, 6, 11, 3, 0, 6, 0, 4, 6, -1, -1, -1, -1, -1, -1, -1},
    {8, 6, 11, 8, 4, 6, 9, 0, 1, -1, -1, -1, -1, -1, -1, -1},
    {9, 4, 6, 9, 6, 3, 9, 3, 1, 11, 3, 6, -1, -1, -1, -1},
    {6, 8, 4, 6, 11, 8, 2, 10, 1, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 10, 3, 0, 11, 0, 6, 11, 0, 4, 6, -1, -1, -1, -1},
    {4, 11, 8, 4, 6, 11, 0, 2, 9, 2, 10, 9, -1, -1, -1, -1},
    {10, 9, 3, 10, 3, 2, 9, 4, 3, 11, 3, 6, 4, 6, 3, -1},
    {8, 2, 3, 8, 4, 2, 4, 6, 2, -1, -1, -1, -1, -1, -1, -1},
    {0, 4, 2, 4, 6, 2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 9, 0, 2, 3, 4, 2, 4, 6, 4, 3, 8, -1, -1, -1, -1},
    {1, 9, 4, 1, 4, 2, 2, 4, 6, -1, -1, -1, -1, -1, -1, -1},
    {8, 1, 3, 8, 6, 1, 8, 4, 6, 6, 10, 1, -1, -1, -1, -1},
    {10, 1, 0, 10, 0, 6, 6, 0, 4, -1, -1, -1, -1, -1, -1, -1},
    {4, 6, 3, 4, 3, 8, 6, 10, 3, 0, 3, 9, 10, 9, 3, -1},
    {10, 9, 4, 6, 10, 4, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 9, 5, 7, 6, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 3, 4, 9, 5, 11, 7, 6, -1, -1, -1, -1, -1, -1, -1},
    {5, 0, 1, 5, 4, 0, 7, 6, 11, -1, -1, -1, -1, -1, -1, -1},
    {11, 7, 6, 8, 3, 4, 3, 5, 4, 3, 1, 5, -1, -1, -1, -1},
    {9, 5, 4, 10, 1, 2, 7, 6, 11, -1, -1, -1, -1, -1, -1, -1},
    {6, 11, 7, 1, 2, 10, 0, 8, 3, 4, 9, 5, -1, -1, -1, -1},
    {7, 6, 11, 5, 4, 10, 4, 2, 10, 4, 0, 2, -1, -1, -1, -1},
    {3, 4, 8, 3, 5, 4, 3, 2, 5, 10, 5, 2, 11, 7, 6, -1},
    {7, 2, 3, 7, 6, 2, 5, 4, 9, -1, -1, -1, -1, -1, -1, -1},
    {9, 5, 4, 0, 8, 6, 0, 6, 2, 6, 8, 7, -1, -1, -1, -1},
    {3, 6, 2, 3, 7, 6, 1, 5, 0, 5, 4, 0, -1, -1, -1, -1},
    {6, 2, 8, 6, 8, 7, 2, 1, 8, 4, 8, 5, 1, 5, 8, -1},
    {9, 5, 4, 10, 1, 6, 1, 7, 6, 1, 3, 7, -1, -1, -1, -1},
    {1, 6, 10, 1, 7, 6, 1, 0, 7, 8, 7, 0, 9, 5, 4, -1},
    {4, 0, 10, 4, 10, 5, 0, 3, 10, 6, 10, 7, 3, 7, 10, -1},
    {7, 6, 10, 7, 10, 8, 5, 4, 10, 4, 8, 10, -1, -1, -1, -1},
    {6, 9, 5, 6, 11, 9, 11, 8, 9, -1, -1, -1, -1, -1, -1, -1},
    {3, 6, 11, 0, 6, 3, 0, 5, 6, 0, 9, 5, -1, -1, -1, -1},
    {0, 11, 8, 0, 5, 11, 0, 1, 5, 5, 6, 11, -1, -1, -1, -1},
    {6, 11, 3, 6, 3, 5, 5, 3, 1, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 10, 9, 5, 11, 9, 11, 8, 11, 5, 6, -1, -1, -1, -1},
    {0, 11, 3, 0, 6, 11, 0, 9, 6, 5, 6, 9, 1, 2, 10, -1},
    {11, 8, 5, 11, 5, 6, 8, 0, 5, 10, 5, 2, 0, 2, 5, -1},
    {6, 11, 3, 6, 3, 5, 2, 10, 3, 10, 5, 3, -1, -1, -1, -1},
    {5, 8, 9, 5, 2, 8, 5, 6, 2, 3, 8, 2, -1, -1, -1, -1},
    {9, 5, 6, 9, 6, 0, 0, 6, 2, -1, -1, -1, -1, -1, -1, -1},
    {1, 5, 8, 1, 8, 0, 5, 6, 8, 3, 8, 2, 6, 2, 8, -1},
    {1, 5, 6, 2, 1, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 3, 6, 1, 6, 10, 3, 8, 6, 5, 6, 9, 8, 9, 6, -1},
    {10, 1, 0, 10, 0, 6, 9, 5, 0, 5, 6, 0, -1, -1, -1, -1},
    {0, 3, 8, 5, 6, 10, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {10, 5, 6, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {11, 5, 10, 7, 5, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {11, 5, 10, 11, 7, 5, 8, 3, 0, -1, -1, -1, -1, -1, -1, -1},
    {5, 11, 7, 5, 10, 11, 1, 9, 0, -1, -1, -1, -1, -1, -1, -1},
    {10, 7, 5, 10, 11, 7, 9, 8, 1, 8, 3, 1, -1, -1, -1, -1},
    {11, 1, 2, 11, 7, 1, 7, 5, 1, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 3, 1, 2, 7, 1, 7, 5, 7, 2, 11, -1, -1, -1, -1},
    {9, 7, 5, 9, 2, 7, 9, 0, 2, 2, 11, 7, -1, -1, -1, -1},
    {7, 5, 2, 7, 2, 11, 5, 9, 2, 3, 2, 8, 9, 8, 2, -1},
    {2, 5, 10, 2, 3, 5, 3, 7, 5, -1, -1, -1, -1, -1, -1, -1},
    {8, 2, 0, 8, 5, 2, 8, 7, 5, 10, 2, 5, -1, -1, -1, -1},
    {9, 0, 1, 5, 10, 3, 5, 3, 7, 3, 10, 2, -1, -1, -1, -1},
    {9, 8, 2, 9, 2, 1, 8, 7, 2, 10, 2, 5, 7, 5, 2, -1},
    {1, 3, 5, 3, 7, 5, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 7, 0, 7, 1, 1, 7, 5, -1, -1, -1, -1, -1, -1, -1},
    {9, 0, 3, 9, 3, 5, 5, 3, 7, -1, -1, -1, -1, -1, -1, -1},
    {9, 8, 7, 5, 9, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {5, 8, 4, 5, 10, 8, 10, 11, 8, -1, -1, -1, -1, -1, -1, -1},
    {5, 0, 4, 5, 11, 0, 5, 10, 11, 11, 3, 0, -1, -1, -1, -1},
    {0, 1, 9, 8, 4, 10, 8, 10, 11, 10, 4, 5, -1, -1, -1, -1},
    {10, 11, 4, 10, 4, 5, 11, 3, 4, 9, 4, 1, 3, 1, 4, -1},
    {2, 5, 1, 2, 8, 5, 2, 11, 8, 4, 5, 8, -1, -1, -1, -1},
    {0, 4, 11, 0, 11, 3, 4, 5, 11, 2, 11, 1, 5, 1, 11, -1},
    {0, 2, 5, 0, 5, 9, 2, 11, 5, 4, 5, 8, 11, 8, 5, -1},
    {9, 4, 5, 2, 11, 3, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {2, 5, 10, 3, 5, 2, 3, 4, 5, 3, 8, 4, -1, -1, -1, -1},
    {5, 10, 2, 5, 2, 4, 4, 2, 0, -1, -1, -1, -1, -1, -1, -1},
    {3, 10, 2, 3, 5, 10, 3, 8, 5, 4, 5, 8, 0, 1, 9, -1},
    {5, 10, 2, 5, 2, 4, 1, 9, 2, 9, 4, 2, -1, -1, -1, -1},
    {8, 4, 5, 8, 5, 3, 3, 5, 1, -1, -1, -1, -1, -1, -1, -1},
    {0, 4, 5, 1, 0, 5, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {8, 4, 5, 8, 5, 3, 9, 0, 5, 0, 3, 5, -1, -1, -1, -1},
    {9, 4, 5, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 11, 7, 4, 9, 11, 9, 10, 11, -1, -1, -1, -1, -1, -1, -1},
    {0, 8, 3, 4, 9, 7, 9, 11, 7, 9, 10, 11, -1, -1, -1, -1},
    {1, 10, 11, 1, 11, 4, 1, 4, 0, 7, 4, 11, -1, -1, -1, -1},
    {3, 1, 4, 3, 4, 8, 1, 10, 4, 7, 4, 11, 10, 11, 4, -1},
    {4, 11, 7, 9, 11, 4, 9, 2, 11, 9, 1, 2, -1, -1, -1, -1},
    {9, 7, 4, 9, 11, 7, 9, 1, 11, 2, 11, 1, 0, 8, 3, -1},
    {11, 7, 4, 11, 4, 2, 2, 4, 0, -1, -1, -1, -1, -1, -1, -1},
    {11, 7, 4, 11, 4, 2, 8, 3, 4, 3, 2, 4, -1, -1, -1, -1},
    {2, 9, 10, 2, 7, 9, 2, 3, 7, 7, 4, 9, -1, -1, -1, -1},
    {9, 10, 7, 9, 7, 4, 10, 2, 7, 8, 7, 0, 2, 0, 7, -1},
    {3, 7, 10, 3, 10, 2, 7, 4, 10, 1, 10, 0, 4, 0, 10, -1},
    {1, 10, 2, 8, 7, 4, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 9, 1, 4, 1, 7, 7, 1, 3, -1, -1, -1, -1, -1, -1, -1},
    {4, 9, 1, 4, 1, 7, 0, 8, 1, 8, 7, 1, -1, -1, -1, -1},
    {4, 0, 3, 7, 4, 3, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {4, 8, 7, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {9, 10, 8, 10, 11, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {3, 0, 9, 3, 9, 11, 11, 9, 10, -1, -1, -1, -1, -1, -1, -1},
    {0, 1, 10, 0, 10, 8, 8, 10, 11, -1, -1, -1, -1, -1, -1, -1},
    {3, 1, 10, 11, 3, 10, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 2, 11, 1, 11, 9, 9, 11, 8, -1, -1, -1, -1, -1, -1, -1},
    {3, 0, 9, 3, 9, 11, 1, 2, 9, 2, 11, 9, -1, -1, -1, -1},
    {0, 2, 11, 8, 0, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {3, 2, 11, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {2, 3, 8, 2, 8, 10, 10, 8, 9, -1, -1, -1, -1, -1, -1, -1},
    {9, 10, 2, 0, 9, 2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {2, 3, 8, 2, 8, 10, 0, 1, 8, 1, 10, 8, -1, -1, -1, -1},
    {1, 10, 2, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {1, 3, 8, 9, 1, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 9, 1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {0, 3, 8, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
    {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1},
};

// The polygons of every case from the cube geometry, checked against the
// triangle lists above.  On each face the crossing edges pair up into
// segments (an ambiguous face cuts off its two corners above the iso value);
// segments are oriented so that, looking at the face from outside with its
// corners counter-clockwise, a segment starts at the crossing entered from a
// corner below the iso value.  The triangles of a case must cover exactly the
// polygons these segments close into, with the same orientation: their
// directed boundary edges (those whose reverse is not an edge of another
// triangle) are the segments.  Returns false if any case disagrees.
bool mc_tables_host(int* edge_table, signed char* tri_table) {
    int face[6][4];
    int nf = 0;
    for (int axis = 0; axis < 3; ++axis)
        for (int val = 0; val < 2; ++val) {
            int cs[4], k = 0;
            for (int c = 0; c < 8; ++c)
                if (kCorner[c][axis] == val) cs[k++] = c;
            int o[4] = {cs[0], -1, -1, -1};
            for (int i = 1; i < 4; ++i)
                for (int j = 0; j < 4; ++j) {
                    int c = cs[j];
                    bool used = false;
                    for (int u = 0; u < i; ++u) used |= (o[u] == c);
                    int dist = 0;
                    for (int d = 0; d < 3; ++d) dist += abs(kCorner[c][d] - kCorner[o[i - 1]][d]);
                    if (!used && dist == 1) {
                        o[i] = c;
                        break;
                    }
                }
            // (o1 - o0) x (o2 - o1) must point along the outward normal
            int a[3], b[3];
            for (int d = 0; d < 3; ++d) {
                a[d] = kCorner[o[1]][d] - kCorner[o[0]][d];
                b[d] = kCorner[o[2]][d] - kCorner[o[1]][d];
            }
            int cr[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
            if (cr[axis] * (val ? 1 : -1) < 0) {
                int tmp = o[1];
                o[1] = o[3];
                o[3] = tmp;
            }
            for (int i = 0; i < 4; ++i) face[nf][i] = o[i];
            ++nf;
        }
    auto edge_of = [](int p, int q) {
        for (int e = 0; e < 12; ++e)
            if ((edge_a(e) == p && edge_b(e) == q) || (edge_a(e) == q && edge_b(e) == p)) return e;
        return -1;
    };
    bool ok = true;
    for (int ci = 0; ci < 256; ++ci) {
        int above[8];
        for (int c = 0; c < 8; ++c) above[c] = (ci >> c) & 1;
        int mask = 0;
        for (int e = 0; e < 12; ++e)
            if (above[edge_a(e)] != above[edge_b(e)]) mask |= 1 << e;
        edge_table[ci] = mask;
        int next[12];
        for (int e = 0; e < 12; ++e) next[e] = -1;
        for (int f = 0; f < 6; ++f) {
            int ce[4], from_above[4], n = 0;
            for (int k = 0; k < 4; ++k) {
                int p = face[f][k], q = face[f][(k + 1) & 3];
                if (above[p] != above[q]) {
                    ce[n] = edge_of(p, q);
                    from_above[n] = above[p];
                    ++n;
                }
            }
            int seg[2][2], ns = 0;
            if (n == 2) {
                seg[0][0] = 0;
                seg[0][1] = 1;
                ns = 1;
            } else if (n == 4) {
                if (above[face[f][0]]) {
                    seg[0][0] = 3; seg[0][1] = 0;
                    seg[1][0] = 1; seg[1][1] = 2;
                } else {
                    seg[0][0] = 0; seg[0][1] = 1;
                    seg[1][0] = 2; seg[1][1] = 3;
                }
                ns = 2;
            }
            for (int k = 0; k < ns; ++k) {
                int x = seg[k][0], y = seg[k][1];
                if (!from_above[x])
                    next[ce[x]] = ce[y];
                else
                    next[ce[y]] = ce[x];
            }
        }
        // directed edge counts of the case's triangles
        int de[12][12] = {};
        int w = 0;
        for (; w < 16 && kTriangles[ci][w] >= 0; w += 3)
            for (int k = 0; k < 3; ++k) {
                const int p = kTriangles[ci][w + k], q = kTriangles[ci][w + (k + 1) % 3];
                if (p < 0 || p > 11 || q < 0 || q > 11 || !(mask >> p & 1)) ok = false;
                else ++de[p][q];
            }
        for (int p = 0; p < 12; ++p)
            for (int q = 0; q < 12; ++q) {
                const bool boundary = de[p][q] == 1 && de[q][p] == 0;
                const bool interior = de[p][q] == 1 && de[q][p] == 1;
                if (de[p][q] > 1 || (de[p][q] == 1 && !boundary && !interior)) ok = false;
                if (boundary != (next[p] == q)) ok = false;
            }
        for (int k = 0; k < 16; ++k) tri_table[ci * 16 + k] = kTriangles[ci][k];
    }
    return ok;
}

int mc_upload_tables() {
    // once per device; the lock makes concurrent first calls from several host
    // threads upload once and return only after the upload
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    DWG_CHECK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return DWG_OK;
    int et[256];
    signed char tt[256 * 16];
    DWG_REQUIRE(mc_tables_host(et, tt), "marching cubes: a case's triangles do not match its polygons");
    unsigned char nt[256];
    unsigned short es[256];
    for (int i = 0; i < 256; ++i) {
        int k = 0;
        while (k < 16 && tt[i * 16 + k] >= 0) k += 3;
        nt[i] = (unsigned char)(k / 3);
        es[i] = (unsigned short)et[i];
    }
    DWG_CHECK_CUDA(cudaMemcpyToSymbol(c_tri, tt, sizeof(tt)));
    DWG_CHECK_CUDA(cudaMemcpyToSymbol(c_ntri, nt, sizeof(nt)));
    DWG_CHECK_CUDA(cudaMemcpyToSymbol(c_edges, es, sizeof(es)));
    DWG_CHECK_CUDA(cudaMemcpyToSymbol(g_tri, tt, sizeof(tt)));
    DWG_CHECK_CUDA(cudaMemcpyToSymbol(g_ntri, nt, sizeof(nt)));
    if (dev >= 0 && dev < 64) done[dev] = true;
    return DWG_OK;
}

constexpr int kMcThreads = 256;

struct McArgs {
    const float* __restrict__ field;
    const float* __restrict__ pos;
    int rx, ry, rz;
    long long ncell;
    float ox, oy, oz, h;
    int zoff;  // global z index of local sample 0
    float iso;
    const float* iso_dev;
};

__device__ __forceinline__ int mc_case(const McArgs& a, long long cell, int& x, int& y, int& z,
                                       float v[8], float iso) {
    const long long cx = a.rx - 1, cy = a.ry - 1;
    x = (int)(cell % cx);
    long long t = cell / cx;
    y = (int)(t % cy);
    z = (int)(t / cy);
    int ci = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int ox = ((c & 1) != ((c >> 1) & 1)) ? 1 : 0;
        const int oy = (c >> 1) & 1;
        const int oz = (c & 4) ? 0 : 1;
        v[c] = a.field[(long long)(x + ox) + (long long)a.rx * ((long long)(y + oy) + (long long)a.ry * (z + oz))];
        if (v[c] > iso) ci |= 1 << c;
    }
    return ci;
}

__global__ void __launch_bounds__(kMcThreads) k_mc_count(McArgs a, unsigned int* __restrict__ counts) {
    const float iso = a.iso_dev ? *a.iso_dev : a.iso;
    long long cell = (long long)blockIdx.x * kMcThreads + threadIdx.x;
    unsigned n = 0;
    if (cell < a.ncell) {
        int x, y, z;
        float v[8];
        n = c_ntri[mc_case(a, cell, x, y, z, v, iso)];
    }
    typedef cub::BlockReduce<unsigned, kMcThreads> BR;
    __shared__ typename BR::TempStorage tmp;
    unsigned tot = BR(tmp).Sum(n);
    if (threadIdx.x == 0) counts[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kMcThreads)
    k_mc_emit_cells(McArgs a, const unsigned int* __restrict__ offs, long long cap, float* __restrict__ tris,
              float* __restrict__ cen, float* __restrict__ nrm,
                    long long nb, const unsigned int* __restrict__ counts, unsigned long long* __restrict__ total) {
    const float iso = a.iso_dev ? *a.iso_dev : a.iso;
    if (total && blockIdx.x == 0 && threadIdx.x == 0) *total = (unsigned long long)offs[nb - 1] + counts[nb - 1];
    long long cell = (long long)blockIdx.x * kMcThreads + threadIdx.x;
    int x = 0, y = 0, z = 0, ci = 0;
    float v[8];
    unsigned n = 0;
    if (cell < a.ncell) {
        ci = mc_case(a, cell, x, y, z, v, iso);
        n = c_ntri[ci];
    }
    typedef cub::BlockScan<unsigned, kMcThreads> BS;
    __shared__ typename BS::TempStorage tmp;
    unsigned local;
    BS(tmp).ExclusiveSum(n, local);
    if (!n) return;
    unsigned long long base = (unsigned long long)offs[blockIdx.x] + local;
    float p[8][3];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int ox = ((c & 1) != ((c >> 1) & 1)) ? 1 : 0;
        const int oy = (c >> 1) & 1;
        const int oz = (c & 4) ? 0 : 1;
        const int gx = x + ox, gy = y + oy, gz = z + oz;
        if (a.pos) {
            long long gi = (long long)gx + (long long)a.rx * ((long long)gy + (long long)a.ry * gz);
            p[c][0] = a.pos[gi * 3];
            p[c][1] = a.pos[gi * 3 + 1];
            p[c][2] = a.pos[gi * 3 + 2];
        } else {
            p[c][0] = __fadd_rn(a.ox, __fmul_rn((float)gx, a.h));
            p[c][1] = __fadd_rn(a.oy, __fmul_rn((float)gy, a.h));
            p[c][2] = __fadd_rn(a.oz, __fmul_rn((float)(gz + a.zoff), a.h));
        }
    }
    const unsigned emask = c_edges[ci];
    float vl[12][3];
#pragma unroll
    for (int e = 0; e < 12; ++e) {
        if (!(emask & (1u << e))) continue;
        const int ia = e & 7;
        const int ib = e < 4 ? ((e + 1) & 3) : (e < 8 ? 4 + ((e - 3) & 3) : e - 4);
        float num = __fsub_rn(v[ia], iso);
        float den = __double2float_rn(__dadd_rn((double)__fsub_rn(v[ib], v[ia]), 1e-10));
        float ell = __fdiv_rn(num, den);
#pragma unroll
        for (int d = 0; d < 3; ++d) vl[e][d] = __fsub_rn(p[ia][d], __fmul_rn(ell, __fsub_rn(p[ib][d], p[ia][d])));
    }
    for (unsigned k = 0; k < n; ++k) {
        unsigned long long t = base + k;
        if ((long long)t >= cap) break;
        const int e0 = c_tri[ci][3 * k], e1 = c_tri[ci][3 * k + 1], e2 = c_tri[ci][3 * k + 2];
        float P0[3], P1[3], P2[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            P0[d] = vl[e0][d];
            P1[d] = vl[e1][d];
            P2[d] = vl[e2][d];
        }
        if (tris) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                tris[t * 9 + d] = P0[d];
                tris[t * 9 + 3 + d] = P1[d];
                tris[t * 9 + 6 + d] = P2[d];
            }
        }
        if (cen) {
#pragma unroll
            for (int d = 0; d < 3; ++d) cen[t * 3 + d] = __fdiv_rn(__fadd_rn(__fadd_rn(P0[d], P1[d]), P2[d]), 3.0f);
        }
        if (nrm) {
            float u[3], w[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                u[d] = __fsub_rn(P1[d], P0[d]);
                w[d] = __fsub_rn(P2[d], P0[d]);
            }
            float cx = __fsub_rn(__fmul_rn(u[1], w[2]), __fmul_rn(u[2], w[1]));
            float cy = __fsub_rn(__fmul_rn(u[2], w[0]), __fmul_rn(u[0], w[2]));
            float cz = __fsub_rn(__fmul_rn(u[0], w[1]), __fmul_rn(u[1], w[0]));
            float sc = -inv_len_eps(__fsqrt_rn(sq3_rn(cx, cy, cz)));
            nrm[t * 3] = __fmul_rn(cx, sc);
            nrm[t * 3 + 1] = __fmul_rn(cy, sc);
            nrm[t * 3 + 2] = __fmul_rn(cz, sc);
        }
    }
}

// Grids with rows of kMcThinRow cells and more, and more than kMcFewCells: rows are cut into segments of
// 31 cells (the 32 samples of a warp's lanes), eight consecutive segments (in
// cell order) are a unit of the output.
//
// Count: a warp marches a segment kMcMarch rows in y.  The comparisons of a
// row of samples are one ballot, rows z and z + 1 are kept for the next step,
// and four steps' rows are loaded ahead; a cell's case is eight bits of the
// four row masks.  The field is read once from HBM (the rows shared by
// neighbouring z come from L1: the block's warps are consecutive in z).
constexpr int kMcSeg = 31;
constexpr int kMcUnit = 8;
constexpr int kMcMarch = 16;
constexpr int kMcAhead = 4;
// below, lanes of a segment would idle: a thread per cell in both passes
constexpr int kMcThinRow = 16;
// so do grids of up to as many cells: their units are a few hundred, and a warp
// takes a unit's triangles in turn while most of the GPU idles (whole calls by
// rows and by cells, us, a surface and noise: 40^3 60 and 94, 56 and 69; 48^3 60
// and 84, 56 and 80; 64^3 63 and 95, 70 and 132)
constexpr long long kMcFewCells = 1 << 17;

// case of the cell at each lane from the masks of its rows (z, y), (z, y + 1),
// (z + 1, y), (z + 1, y + 1)
__device__ __forceinline__ unsigned mc_case_bits(unsigned A, unsigned B, unsigned C, unsigned D, int lane) {
    const unsigned b = B >> lane, d = D >> lane;
    return ((C >> lane) & 3u) | (((d & 1u) << 3) | ((d & 2u) << 1)) | (((A >> lane) & 3u) << 4) |
           (((b & 1u) << 7) | ((b & 2u) << 5));
}

__global__ void __launch_bounds__(kMcThreads) k_mc_count_rows(McArgs a, int segs, unsigned int* __restrict__ counts) {
    static_assert(kMcThreads == 256, "a case per thread");
    __shared__ unsigned char ntri[256];
    ntri[threadIdx.x] = g_ntri[threadIdx.x];
    __syncthreads();
    const unsigned FULL = 0xffffffffu;
    const float iso = a.iso_dev ? *a.iso_dev : a.iso;
    const int lane = threadIdx.x & 31;
    const int cx = a.rx - 1, cy = a.ry - 1, cz = a.rz - 1;
    const long long item = ((long long)blockIdx.x * kMcThreads + threadIdx.x) >> 5;
    const int z = (int)(item % cz);
    const long long r = item / cz;
    const int seg = (int)(r % segs), x0 = seg * kMcSeg, y0 = (int)(r / segs) * kMcMarch;
    if (y0 >= cy) return;
    const int y1 = min(y0 + kMcMarch, cy);
    const int last = min(kMcSeg, cx - x0);  // the segment's last sample
    const bool in = lane <= last;
    const unsigned valid = 0xffffffffu >> (31 - last);
    const size_t plane = (size_t)a.rx * a.ry;
    const float* row = a.field + (size_t)z * plane + (size_t)y0 * a.rx + x0 + lane;
    unsigned A = __ballot_sync(FULL, in && row[0] > iso), C = __ballot_sync(FULL, in && row[plane] > iso);
    for (int y = y0; y < y1; y += kMcAhead) {
        float v0[kMcAhead], v1[kMcAhead];
#pragma unroll
        for (int u = 0; u < kMcAhead; ++u) {
            row += a.rx;
            const bool ok = in && y + u < y1;
            v0[u] = ok ? row[0] : 0.f;
            v1[u] = ok ? row[plane] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kMcAhead; ++u) {
            if (y + u >= y1) break;
            const unsigned B = __ballot_sync(FULL, in && v0[u] > iso), D = __ballot_sync(FULL, in && v1[u] > iso);
            if ((A | B | C | D) && (A & B & C & D) != valid) {
                const unsigned n = __reduce_add_sync(FULL, lane < last ? ntri[mc_case_bits(A, B, C, D, lane)] : 0u);
                if (lane == 0 && n)
                    atomicAdd(&counts[(seg + (long long)segs * (y + u + (long long)cy * z)) / kMcUnit], n);
            }
            A = B;
            C = D;
        }
    }
}

// Emit: a warp per unit that has triangles (group units at a time are looked
// at for one).  It finds the cases again by row masks and lists the triangles
// (case, cell, number, segment) in shared memory; 32 of them at a time, a lane
// makes one each from the six samples of its edges (L1), and the vertices
// leave through shared memory as whole rows.  The triangles of consecutive
// units are consecutive in the output, so what does not fill the lanes waits
// for the next unit of the group.  Lanes are busy with triangles, not cells,
// nothing is indexed in local memory, and stores are coalesced.  Also writes
// the total.  A 384^3 grid with 2.05 M triangles: count 109 and emit 257 us (367
// and 897 with a thread per cell in both passes); 256^3 at 0.3 M: 30 and 71
// (91 and 190).  The instructions of the triangles bound it (0.65 of issue).
constexpr int kMcEmitWarps = 4;
constexpr int kMcGroup = 4;                       // units a warp takes at a time, at most
constexpr int kMcPlaces = kMcGroup * kMcUnit;     // segments whose places are kept
constexpr int kMcList = 32 + 5 * kMcSeg;          // waiting triangles, and a segment's

template <bool POS>
__global__ void __launch_bounds__(kMcEmitWarps * 32)
    k_mc_emit(McArgs a, unsigned segs, const unsigned int* __restrict__ counts, const unsigned int* __restrict__ offs,
              long long units, int group, long long cap, float* __restrict__ tris, float* __restrict__ cen,
              float* __restrict__ nrm, unsigned long long* __restrict__ total) {
    __shared__ __align__(16) signed char edges[256][16];
    __shared__ unsigned char ntri[256];
    __shared__ size_t corner[8];
    // case | lane << 8 | number << 13 | segment << 16
    __shared__ unsigned list[kMcEmitWarps][kMcList];
    __shared__ int3 place[kMcEmitWarps][kMcPlaces];  // x0, y, z of the listed segments
    __shared__ float out[kMcEmitWarps][32 * 9];
    for (int i = threadIdx.x; i < 256; i += kMcEmitWarps * 32) {
        *reinterpret_cast<int4*>(edges[i]) = *reinterpret_cast<const int4*>(g_tri[i]);
        ntri[i] = g_ntri[i];
    }
    const size_t plane = (size_t)a.rx * a.ry;
    if (threadIdx.x < 8) {
        const int c = threadIdx.x;
        corner[c] = ((c ^ (c >> 1)) & 1) + (size_t)((c >> 1) & 1) * a.rx + (size_t)(1 - (c >> 2)) * plane;
    }
    __syncthreads();
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const float iso = a.iso_dev ? *a.iso_dev : a.iso;
    const int cx = a.rx - 1;
    const unsigned cy = (unsigned)(a.ry - 1), cz = (unsigned)(a.rz - 1);
    if (total && blockIdx.x == 0 && threadIdx.x == 0)
        *total = (unsigned long long)offs[units - 1] + counts[units - 1];
    // the listed triangles first .. first + n - 1 go to dst rows (width floats)
    auto store = [&](float* dst, int width, int m, unsigned long long at) {
        __syncwarp();
        float* o = dst + at * width;
        for (int k = lane; k < m * width; k += 32) o[k] = out[w][k];
        __syncwarp();
    };
    auto emit = [&](int n, unsigned long long at) {  // the list's first n (1 to 32) triangles
        const long long left = cap - (long long)at;  // that still fit
        if (left <= 0) return;
        const int m = left < n ? (int)left : n;
        float P[3][3];
        if (lane < m) {
            const unsigned en = list[w][lane];
            const int3 o = place[w][en >> 16];
            const int x = o.x + (int)((en >> 8) & 31u), y = o.y, z = o.z;
            const signed char* tri = &edges[en & 255u][3 * ((en >> 13) & 7u)];
            const float* f = a.field + ((size_t)x + (size_t)a.rx * y + plane * z);
            // the cell's coordinates on each axis
            const float x0 = __fadd_rn(a.ox, __fmul_rn((float)x, a.h)), x1 = __fadd_rn(a.ox, __fmul_rn((float)(x + 1), a.h));
            const float y0 = __fadd_rn(a.oy, __fmul_rn((float)y, a.h)), y1 = __fadd_rn(a.oy, __fmul_rn((float)(y + 1), a.h));
            const int gz = z + a.zoff;
            const float z0 = __fadd_rn(a.oz, __fmul_rn((float)gz, a.h)), z1 = __fadd_rn(a.oz, __fmul_rn((float)(gz + 1), a.h));
            int ca[3], cb[3];
            float va[3], vb[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int e = tri[q];
                ca[q] = e & 7;
                cb[q] = e < 4 ? ((e + 1) & 3) : (e < 8 ? 4 + ((e - 3) & 3) : e - 4);
                va[q] = f[corner[ca[q]]];
                vb[q] = f[corner[cb[q]]];
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float num = __fsub_rn(va[q], iso);
                const float den = __double2float_rn(__dadd_rn((double)__fsub_rn(vb[q], va[q]), 1e-10));
                const float ell = __fdiv_rn(num, den);
                float p[2][3];
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int c = s ? cb[q] : ca[q];
                    if (POS) {
                        const float* r = a.pos + 3 * ((f - a.field) + corner[c]);
                        p[s][0] = r[0];
                        p[s][1] = r[1];
                        p[s][2] = r[2];
                    } else {
                        p[s][0] = (c ^ (c >> 1)) & 1 ? x1 : x0;
                        p[s][1] = c & 2 ? y1 : y0;
                        p[s][2] = c & 4 ? z0 : z1;
                    }
                }
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    P[q][d] = __fsub_rn(p[0][d], __fmul_rn(ell, __fsub_rn(p[1][d], p[0][d])));
            }
        }
        if (tris) {
            if (lane < m) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) out[w][lane * 9 + q * 3 + d] = P[q][d];
            }
            store(tris, 9, m, at);
        }
        if (cen) {
            if (lane < m) {
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    out[w][lane * 3 + d] = __fdiv_rn(__fadd_rn(__fadd_rn(P[0][d], P[1][d]), P[2][d]), 3.0f);
            }
            store(cen, 3, m, at);
        }
        if (nrm) {
            if (lane < m) {
                float u[3], v[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    u[d] = __fsub_rn(P[1][d], P[0][d]);
                    v[d] = __fsub_rn(P[2][d], P[0][d]);
                }
                const float nx = __fsub_rn(__fmul_rn(u[1], v[2]), __fmul_rn(u[2], v[1]));
                const float ny = __fsub_rn(__fmul_rn(u[2], v[0]), __fmul_rn(u[0], v[2]));
                const float nz = __fsub_rn(__fmul_rn(u[0], v[1]), __fmul_rn(u[1], v[0]));
                const float sc = -inv_len_eps(__fsqrt_rn(sq3_rn(nx, ny, nz)));
                out[w][lane * 3] = __fmul_rn(nx, sc);
                out[w][lane * 3 + 1] = __fmul_rn(ny, sc);
                out[w][lane * 3 + 2] = __fmul_rn(nz, sc);
            }
            store(nrm, 3, m, at);
        }
    };
    const long long warps = (long long)gridDim.x * kMcEmitWarps;
    for (long long g = (long long)blockIdx.x * kMcEmitWarps + w; g * group < units; g += warps) {
        const long long mine = g * group + lane;
        const unsigned cnt = lane < group && mine < units ? counts[mine] : 0u;
        unsigned act = __ballot_sync(FULL, cnt > 0);
        if (!act) continue;
        unsigned long long base = offs[g * group + __ffs(act) - 1];  // output place of the list's first triangle
        int T = 0, ns = 0;                                           // triangles waiting, segments placed
        while (act) {
            const long long unit = g * group + __ffs(act) - 1;
            act &= act - 1;
            // lane s: the place of the unit's segment s (of a lane past the
            // grid's segments, z = cz)
            const unsigned seg = (unsigned)unit * kMcUnit + (lane & (kMcUnit - 1));
            const unsigned st = seg / segs;
            const int sx = (int)(seg - st * segs) * kMcSeg;
            const unsigned sz = st / cy, sy = st - sz * cy;
            if (lane < kMcUnit) place[w][ns + lane] = make_int3(sx, (int)sy, (int)sz);
            // the cases of the unit's cells, a byte per segment
            unsigned long long ci8 = 0;
#pragma unroll
            for (int s = 0; s < kMcUnit; ++s) {
                const int x = __shfl_sync(FULL, sx, s) + lane;
                const unsigned y = __shfl_sync(FULL, sy, s), z = __shfl_sync(FULL, sz, s);
                bool va = false, vb = false, vc = false, vd = false;
                if (x < a.rx && z < cz) {
                    const float* p = a.field + (size_t)x + (size_t)a.rx * y + plane * z;
                    va = p[0] > iso;
                    vb = p[a.rx] > iso;
                    vc = p[plane] > iso;
                    vd = p[plane + a.rx] > iso;
                }
                const unsigned A = __ballot_sync(FULL, va), B = __ballot_sync(FULL, vb), C = __ballot_sync(FULL, vc),
                               D = __ballot_sync(FULL, vd);
                if (lane < kMcSeg && x < cx) ci8 |= (unsigned long long)mc_case_bits(A, B, C, D, lane) << (8 * s);
            }
            // (after the group's last unit, once more for what waits)
#pragma unroll 1
            for (int s = 0; s < kMcUnit + (act ? 0 : 1); ++s) {
                if (s < kMcUnit) {
                    const unsigned ci = (unsigned)(ci8 >> (8 * s)) & 255u;
                    const int n = ntri[ci];
                    // n is at most 5: three ballots count the triangles before
                    const unsigned b0 = __ballot_sync(FULL, n & 1), b1 = __ballot_sync(FULL, n & 2),
                                   b2 = __ballot_sync(FULL, n & 4);
                    if (!(b0 | b1 | b2)) continue;
                    const int at = T + __popc(b0 & below) + 2 * __popc(b1 & below) + 4 * __popc(b2 & below);
                    for (int k = 0; k < n; ++k) list[w][at + k] = ci | (lane << 8) | (k << 13) | ((ns + s) << 16);
                    T += __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
                }
                while (T >= 32 || (s == kMcUnit && T > 0)) {
                    __syncwarp();
                    const int m = min(T, 32);
                    emit(m, base);
                    base += m;
                    T -= m;
                    __syncwarp();
                    // the others move up (in order: a row of lanes at a time)
                    for (int k = 0; k < T; k += 32) {
                        const unsigned v = k + lane < T ? list[w][k + 32 + lane] : 0u;
                        __syncwarp();
                        if (k + lane < T) list[w][k + lane] = v;
                        __syncwarp();
                    }
                }
            }
            ns += kMcUnit;
        }
    }
}

// how a grid is cut: blocks of cells (segs 0) or units of segments
struct McCut {
    unsigned segs;
    long long parts;
};
static McCut mc_cut(const McArgs& a, long long most_parts) {
    const long long cx = a.rx - 1, rows = (long long)(a.ry - 1) * (a.rz - 1);
    const long long segs = (cx + kMcSeg - 1) / kMcSeg, units = (segs * rows + kMcUnit - 1) / kMcUnit;
    if (cx >= kMcThinRow && a.ncell > kMcFewCells && segs * rows < (1ll << 32) - kMcUnit && units <= most_parts)
        return {(unsigned)segs, units};
    return {0u, (a.ncell + kMcThreads - 1) / kMcThreads};
}

// triangles per part of the grid
static int mc_count(const McArgs& a, const McCut& cut, unsigned int* counts, cudaStream_t s) {
    if (cut.segs) {
        const long long marches = (a.ry - 1 + kMcMarch - 1) / kMcMarch;
        const long long blocks = ((long long)cut.segs * marches * (a.rz - 1) * 32 + kMcThreads - 1) / kMcThreads;
        DWG_CHECK_CUDA(cudaMemsetAsync(counts, 0, sizeof(unsigned int) * cut.parts, s));
        k_mc_count_rows<<<(unsigned)blocks, kMcThreads, 0, s>>>(a, (int)cut.segs, counts);
    } else {
        k_mc_count<<<(unsigned)cut.parts, kMcThreads, 0, s>>>(a, counts);
    }
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

// the triangles at their offsets, and (total not null) their number
static int mc_emit(const McArgs& a, const McCut& cut, const unsigned int* counts, const unsigned int* offs,
                   long long cap, float* tris, float* centroids, float* normals, unsigned long long* total,
                   cudaStream_t s) {
    if (cut.segs) {
        static int bps_of[2] = {0, 0};
        int& bps = bps_of[a.pos != nullptr];
        if (!bps) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, a.pos ? k_mc_emit<true> : k_mc_emit<false>,
                                                          kMcEmitWarps * 32, 0);
            if (bps <= 0) bps = 1;
        }
        // several groups per warp, so that clusters of units with triangles
        // spread over the warps
        const long long warps = (long long)num_sms() * bps * kMcEmitWarps;
        const int group = (int)std::max<long long>(1, std::min<long long>(kMcGroup, cut.parts / (4 * warps)));
        const long long blocks = std::min<long long>((long long)num_sms() * bps,
                                                     (cut.parts + (long long)group * kMcEmitWarps - 1) /
                                                         ((long long)group * kMcEmitWarps));
        auto kernel = a.pos ? k_mc_emit<true> : k_mc_emit<false>;
        kernel<<<(unsigned)blocks, kMcEmitWarps * 32, 0, s>>>(a, cut.segs, counts, offs, cut.parts, group, cap, tris,
                                                              centroids, normals, total);
    } else {
        k_mc_emit_cells<<<(unsigned)cut.parts, kMcThreads, 0, s>>>(a, offs, cap, tris, centroids, normals, cut.parts,
                                                                   counts, total);
    }
    DWG_CHECK_LAUNCH();
    return DWG_OK;
}

int mc_run(const float* field, const McGrid& g, float iso, const float* iso_dev, float* tris,
           float* centroids, float* normals, long long cap, unsigned long long* num_tris_dev,
           McWorkspace& ws, cudaStream_t s) {
    DWG_REQUIRE(field && num_tris_dev, "marching cubes: null field or count pointer");
    DWG_REQUIRE(g.res[0] >= 2 && g.res[1] >= 2 && g.res[2] >= 2, "marching cubes: resolution must be >= 2");
    DWG_TRY(mc_upload_tables());
    McArgs a;
    a.field = field;
    a.pos = g.positions;
    a.rx = g.res[0];
    a.ry = g.res[1];
    a.rz = g.res[2];
    a.ncell = (long long)(g.res[0] - 1) * (g.res[1] - 1) * (g.res[2] - 1);
    a.ox = g.origin[0];
    a.oy = g.origin[1];
    a.oz = g.origin[2];
    a.zoff = g.zoff;
    a.h = g.spacing;
    a.iso = iso;
    a.iso_dev = iso_dev;
    DWG_REQUIRE((a.ncell + kMcThreads - 1) / kMcThreads < (1ll << 31), "marching cubes: grid too large");
    const McCut cut = mc_cut(a, 1ll << 30);
    const long long nb = cut.parts;
    DWG_TRY(ws.block_counts.reserve(nb));
    DWG_TRY(ws.block_offsets.reserve(nb));
    DWG_TRY(mc_count(a, cut, ws.block_counts.ptr, s));
    size_t bytes = 0;
    unsigned* cin = ws.block_counts.ptr;
    unsigned* cout = ws.block_offsets.ptr;
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, cin, cout, (int)nb, s));
    DWG_TRY(ws.scratch.reserve(bytes + 256));
    bytes = ws.scratch.n;
    DWG_CHECK_CUDA(cub::DeviceScan::ExclusiveSum(ws.scratch.ptr, bytes, cin, cout, (int)nb, s));
    return mc_emit(a, cut, cin, cout, cap, tris, centroids, normals, num_tris_dev, s);
}

}  // namespace dwg

// ----------------------------------------------------------------------------
// Marching cubes without any device allocation.
//
// Some callers cannot call cudaMalloc when they mesh: a real-time loop that
// must not allocate after start-up (cudaMalloc and cudaFree can wait for the
// whole device), or an application whose device memory is a fixed budget
// handed out by its own pool.  dwg_marching_cubes_noalloc serves them with the
// same two kernels as dwg_marching_cubes; its scratch (per-block triangle
// counts, their offsets and the total) lives in the file-scope device array
// below, which every GPU that loads this library holds until the process
// exits.  The scan writes every offset and the total it later reads, so
// nothing has to be cleared between calls.
// ----------------------------------------------------------------------------
namespace dwg {

// 2^19 blocks of 256 cells: grids up to 134,217,728 cells (e.g. 512^3)
constexpr long long kMcNoAllocMaxBlocks = 1ll << 19;
constexpr long long kMcNoAllocMaxCells = kMcNoAllocMaxBlocks * kMcThreads;
// [0, max) block counts, [max, 2 max) block offsets, then the 64-bit total
static __device__ __align__(256) unsigned int g_mc_noalloc_scratch[2 * kMcNoAllocMaxBlocks + 64];

// exclusive scan of the block counts by one block, in chunks, with a carry;
// writes every offset and the total, so no slot has to start at zero
constexpr int kMcScanThreads = 1024;
__global__ void __launch_bounds__(kMcScanThreads)
    k_mc_noalloc_scan(const unsigned int* __restrict__ counts, unsigned int* __restrict__ offs, long long nb,
                      unsigned long long* __restrict__ total) {
    typedef cub::BlockScan<unsigned long long, kMcScanThreads> BS;
    __shared__ typename BS::TempStorage tmp;
    __shared__ unsigned long long carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (long long base = 0; base < nb; base += kMcScanThreads) {
        const long long i = base + threadIdx.x;
        const unsigned long long v = i < nb ? counts[i] : 0ull;
        unsigned long long ex, agg;
        BS(tmp).ExclusiveSum(v, ex, agg);
        if (i < nb) offs[i] = (unsigned int)(carry + ex);
        __syncthreads();
        if (threadIdx.x == 0) carry += agg;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// device address of the scratch array, looked up once per device with that
// device current (the host-side symbol is not a device address)
static int mc_noalloc_scratch(unsigned int** out) {
    static std::mutex mu;
    static unsigned int* addr[64] = {nullptr};
    int dev = 0;
    DWG_CHECK_CUDA(cudaGetDevice(&dev));
    DWG_REQUIRE(dev >= 0 && dev < 64, "marching_cubes_noalloc: device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_mc_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            set_error("marching_cubes_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return DWG_ERR_CUDA;
        }
        addr[dev] = (unsigned int*)p;
    }
    *out = addr[dev];
    return DWG_OK;
}

}  // namespace dwg

extern "C" int dwg_marching_cubes_noalloc(const float* field_dev, const int res[3], const float* positions_dev,
                                          const float origin[3], float spacing, float iso, float* tris_dev,
                                          float* centroids_dev, float* normals_dev, long long capacity,
                                          long long* num_tris_host, void* stream) {
    using namespace dwg;
    DWG_REQUIRE(field_dev && res && num_tris_host, "marching_cubes_noalloc: null field, resolution or count");
    DWG_REQUIRE(origin || positions_dev, "marching_cubes_noalloc: grid undefined (no origin, no positions)");
    DWG_REQUIRE(res[0] >= 2 && res[1] >= 2 && res[2] >= 2, "marching_cubes_noalloc: resolution must be >= 2");
    DWG_REQUIRE(capacity >= 0, "marching_cubes_noalloc: negative capacity");
    const long long ncell = (long long)(res[0] - 1) * (res[1] - 1) * (res[2] - 1);
    DWG_REQUIRE(ncell <= kMcNoAllocMaxCells,
                "marching_cubes_noalloc: %lld cells exceed the allocation-free limit of %lld cells; use "
                "dwg_marching_cubes",
                ncell, kMcNoAllocMaxCells);
    DWG_TRY(mc_upload_tables());
    unsigned int* scratch = nullptr;
    DWG_TRY(mc_noalloc_scratch(&scratch));
    unsigned int* counts = scratch;
    unsigned int* offs = scratch + kMcNoAllocMaxBlocks;
    unsigned long long* total = reinterpret_cast<unsigned long long*>(scratch + 2 * kMcNoAllocMaxBlocks);
    cudaStream_t s = (cudaStream_t)stream;
    McArgs a;
    a.field = field_dev;
    a.pos = positions_dev;
    a.rx = res[0];
    a.ry = res[1];
    a.rz = res[2];
    a.ncell = ncell;
    a.ox = origin ? origin[0] : 0.f;
    a.oy = origin ? origin[1] : 0.f;
    a.oz = origin ? origin[2] : 0.f;
    a.zoff = 0;
    a.h = spacing;
    a.iso = iso;
    a.iso_dev = nullptr;
    const McCut cut = mc_cut(a, kMcNoAllocMaxBlocks);
    const long long nb = cut.parts;
    DWG_TRY(mc_count(a, cut, counts, s));
    k_mc_noalloc_scan<<<1, kMcScanThreads, 0, s>>>(counts, offs, nb, total);
    DWG_CHECK_LAUNCH();
    DWG_TRY(mc_emit(a, cut, counts, offs, capacity, tris_dev, centroids_dev, normals_dev, nullptr, s));
    unsigned long long T = 0;
    DWG_CHECK_CUDA(cudaMemcpyAsync(&T, total, sizeof(T), cudaMemcpyDeviceToHost, s));
    DWG_CHECK_CUDA(cudaStreamSynchronize(s));
    *num_tris_host = (long long)T;
    if ((long long)T > capacity) {
        set_error("marching_cubes_noalloc: %llu triangles exceed capacity %lld", T, capacity);
        return DWG_ERR_OVERFLOW;
    }
    return DWG_OK;
}
