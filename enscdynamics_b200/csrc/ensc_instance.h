// Host-side preparation and device layout of one solver instance, shared by
// the single-instance handle (ensc_capi.cu) and the batch (ensc_batch.cu).
// Internal; not part of the ABI.
#pragma once

#include "ensc_gpu.h"
#include "ensc_device.cuh"

#include <cuda_runtime.h>

#include <string>
#include <vector>

namespace ensc {

// Everything exDyna3D::init() derives from the deck before stepping
// (Explicit3D/source/exDyna3D.cpp:105-142) that the device needs, in host
// memory, plus the byte layout of the instance's device block.
struct InstanceHost {
    int64_t nn = 0, ne = 0, nn_pad = 0, ne_pad = 0;
    bool mixed = false, plastic = false, clash = false;
    // (bt, jinv and vol0 in the caller's order, and only until the tiles hold them)
    std::vector<double> bt;           // [ne][24] row-major B0^T
    std::vector<double> jinv;         // [ne][9] J^-1 / 8 where bt9
    std::vector<double> vol0;         // [ne] V0
    std::vector<double> im;           // [nn_pad] inverse lumped mass per node
    // clash meshes (a node repeats a local slot): with at most 8 elements at
    // every node, rows of the force array [ne_pad] (ElemArrays::rows) and
    // merge flags [nn_pad] (NodeArrays::merge); else (slot, element)-sorted lists
    std::vector<uint32_t> rows;
    std::vector<uint8_t> merge;
    std::vector<int64_t> csr_ptr;
    std::vector<uint32_t> csr_ent;
    const double* x0 = nullptr;       // caller arrays, read by instance_prepare only
    const double* v0 = nullptr;
    // what the upload copies as it is, formed by instance_prepare (so that a
    // prepared instance's host work is done before its device part): the
    // constant part of every element tile (connectivity, geometry, V0 and its
    // roots), const_bytes each; the node records (NodeArrays) -- FP64: q0, q1 and
    // vz; mixed: q0 with two velocities packed in, vz and the 16-bit residual rows
    // [3][nn_pad] (what only holds velocities stays empty when the mesh has none)
    int32_t tile_bytes = 0, const_bytes = 0;
    bool bt9 = false;                 // FP64: 9 numbers per element give B0^T bit for bit
    std::vector<unsigned char> tiles;
    std::vector<double> q0, q1, vz_d;
    std::vector<float> vz_f;
    std::vector<int16_t> v_lo;
    // element of the caller's numbering -> stored position; empty: the same.
    // Tiles, rows and lists are of stored elements
    std::vector<int32_t> iperm;
    // patch assembly: the patch tables
    bool patch = false;
    std::vector<uint32_t> pf_off;     // [n_patches + 1]
    std::vector<uint32_t> pinc_off;   // [n_pnodes + 1]
    std::vector<uint16_t> pinc;       // [8 ne]
    std::vector<uint32_t> nptr;       // [nn + 1]
    std::vector<uint32_t> nent;       // [n_pnodes]
    int64_t n_patches = 0, n_pnodes = 0;
    // device layout: byte offsets of the pieces in one 256-byte-aligned block
    enum Piece {
        TILES, FE, X, U, V, IM, BC, BCV, RF, ROWS, MERGE, CPTR, CENT,
        IPERM, PFOFF, PINCOFF, PINC, PF, NPTR, NENT, NPIECE
    };
    size_t off[NPIECE] = {};
    size_t size[NPIECE] = {};
    size_t bytes = 0;
};

// Validates the mesh and fills `h` (element constants computed as
// compute_invMassMatrix does unless the caller supplies them).
int instance_prepare(const ensc_mesh_desc* mesh, const ensc_material* mat, bool mixed, int assembly,
                     InstanceHost& h, std::string& err);

// Stored order of the slot assembly, as patch_order; empty: the caller's order.
// Warps gather node records and store forces best where the elements of a tile
// follow the node numbering.  Where a slot's node leaves its group of 4 from one
// element to the next in more than 3 of 8 slots (a block's rows: 2.0 to 2.2), the
// elements are sorted by their nodes; the sorted order is taken where it leaves
// at most 4/5 of the changes.  B200, us a cycle of 196,608 elements (FP64, mixed)
// as given and sorted, a block's element order cut into shuffled runs:
//   changes 8.0   69.8, 56.3   44.4, 30.4        3.0   48.1, 33.2   44.4, 29.8
//           5.0   53.5, 40.7   44.4, 30.2        2.5   46.5, 31.5   44.5, 30.5
//           3.5   48.5, 34.1   44.4, 30.3        2.0   44.3, 30.4   44.5, 30.2
// and with the node numbers shuffled too, within 8, 64 and all of the nodes:
//   8.0, sorted 5.3   71.0, 56.9   45.9, 31.4
//   8.0, sorted 7.4   72.2, 59.2   49.6, 34.1
//   8.0, sorted 8.0   66.4, 53.3   68.9, 57.1
// So the first line lies where sorting still gives 8 to 12%, and the second, left
// on the safe side, keeps an order that sorting may lose to (3 to 7% at the
// last); numberings between 4/5 and 1 stay as given although many would gain.
std::vector<int32_t> local_order(int64_t nn, int64_t ne, const uint32_t* conn);

// Stored order of the patch assembly: elements sorted by the Morton key of
// their centroid's cell on a grid of the smallest element extent per axis,
// so that runs of kPatchElems stored elements are compact clusters.  Returns
// perm[stored position] = element of the caller's numbering.
std::vector<int32_t> patch_order(int64_t ne, const uint32_t* conn, const double* x0);

// Builds the patch tables of h (pf_off, pinc_off, pinc, nptr, nent) for the
// stored connectivity conn [ne][8].
void build_patches(int64_t nn, int64_t ne, const uint32_t* conn, InstanceHost& h);

// The device form of a call's boundary conditions: bc[n] packs the codes of node
// n's components, 2 bits each; bcv[3][nn_pad] holds the prescribed velocities and
// stays empty when no component has one (they are read only where one has).
void pack_bcs(int64_t nn, int64_t nn_pad, const int8_t* dof_code, const double* dof_value, std::vector<uint8_t>& bc,
              std::vector<double>& bcv);

// Copies the instance into `block` (h.bytes bytes, 256-byte aligned) on
// stream `st`, waits for the copies, and fills the array descriptors (PA
// all null under the slot assembly).
int instance_upload(const InstanceHost& h, void* block, cudaStream_t st, ElemArrays& E, NodeArrays& N,
                    PatchArrays& PA, std::string& err);

// Material_elastic::update (Material_elastic.cpp:9-14) plus the controls.
void material_from(const ensc_material* mat, const ensc_params* p, Material& M);

// Initial control block for time 0.
Ctl initial_ctl(const ensc_params* p, const Material& M);

}  // namespace ensc
