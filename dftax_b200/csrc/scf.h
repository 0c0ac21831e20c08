// Internal declarations of the Kohn-Sham SCF around the DF J/K plan (scf.cu,
// onee.cu, xc.cu). Not part of the C ABI (include/dfscf.h).
#pragma once

#include "internal.h"
#include "../../include/dfscf.h"

namespace dfjk {

// Device view of the orbital shells for the one-electron and AO kernels.
struct OrbView {
  ShellView sh;
  const int* out0;      // first spherical (or cartesian) function of each shell
  const double* c2s;    // transformation blocks, one per l (ncart(l) x nout(l), row-major)
  int c2s_off[8];       // offset of l's block in c2s
  int nout[8];          // functions per shell of each l (2l+1, or ncart(l) without cart2sph)
  int nao;
};

// One-electron integrals (onee.cu): S, T and V = -sum_C Z_C <a|1/|r-C||b> as
// nao x nao matrices (symmetric, both triangles written), for the shell pairs
// of the orbital basis.
void launch_one_electron(const Context& c, const OrbView& ov, int nshell, const std::vector<int>& l,
                         int natom, const double* atom_xyz, const double* atom_z, double* S,
                         double* T, double* V, cudaStream_t s);

// Chunks of spatially sorted grid points, each with the orbital shells that
// are not negligible anywhere in its bounding box (xc_chunk)
constexpr int kXcMaxL = 3;   // orbital l the AO kernel evaluates (f)

// What the kernels read about a chunk; the offsets (in doubles) lie within the
// buffers of its group
struct XcChunkInfo {
  int nsig, ldp;             // functions of the chunk, and rounded up to even
  int64_t g0, ng;            // first point and count
  int64_t phi, pc, part;     // AO values (dphi at 3 phi), P block, V slices
  int64_t ao;                // first entry of the compact AO map
};

// A run of chunks whose kernels share their launches: the chunks' AO values,
// gradients and weighted AOs take at most kXcGroupBytes (or one chunk). Chunks
// have a function and 256 points at least, so a group's count stays below 2^16.
constexpr int64_t kXcGroupBytes = (int64_t)256 << 20;
static_assert(kXcGroupBytes / (40 * 256) < 65536, "chunks of a group: a grid dimension");
// Points of a chunk, at most: its 512-point slices are a grid dimension too.
constexpr int64_t kXcMaxChunk = (int64_t)1 << 24;
inline int64_t xc_points(int64_t grid_chunk) {   // of a chunk for a requested size
  return grid_chunk < kXcMaxChunk ? (grid_chunk + 255) / 256 * 256 : kXcMaxChunk;
}
struct XcGroup {
  int first = 0, count = 0;            // chunks
  int max_nsig = 0;
  int e_off = 0, e_cnt[kXcMaxL + 1] = {};   // shell entries, by l
};

struct XcChunks {
  int64_t G = 0;                       // points per chunk (the last may hold fewer)
  std::vector<XcChunkInfo> info;
  std::vector<XcGroup> groups;
  int64_t max_phi = 0, max_pc = 0, max_part = 0, max_points = 0;   // largest group, doubles
  double gemm_flop = 0.0;              // FLOP of one evaluation's two products: sum 4 G nsig^2
  // shell entries (shell, its first compact AO, chunk), by group and l; compact
  // AO -> AO of each chunk; AO -> compact AO or -1 ([chunk][nao]); info
  DevBuf d_e_sh, d_e_out0, d_e_chunk, d_ao_map, d_pos, d_info;
};

// XC on a point grid (xc.cu)
// The groups of one XC evaluation run on up to kXcBranches concurrent branches
// (group k on branch k % branches), each with its own buffers, the context's
// stream of that branch and its own V accumulator, so that one group's kernels
// fill the tails of another's. The accumulators are summed in branch order at
// the end and the energy partials are per chunk, so the result does not depend
// on how the branches interleave.
struct XcBranch {
  DevBuf phi, dphi, W;          // per chunk [nsig][G]: AO values, 3 gradients, weighted AO
  DevBuf Pc, Vc;                // P on each chunk's AOs, the slices of its V block
  DevBuf vals;                  // per chunk [4][G]: rho, grad rho, then v_rho / 2, v_grad
};

// Upper bound of a branch's buffers (its V accumulators too) for chunks of G of
// npoint points and nao functions
int64_t xc_branch_bytes(int64_t nao, int64_t G, int64_t npoint);

// branches of an evaluation unless the caller asks for another number. us by group
// size and branches, 512-point chunks, (H2O)_6 / (H2O)_16 / C8H18: 96 MB x 4 860 /
// 4940 / 5070, 256 x 1 986 / 6130 / 6330, 256 x 2 893 / 5070 / 5130, 256 x 4 821 /
// 4820 / 4800, 256 x 8 836 / 4770 / 4810, 1024 x 4 879 / 4840 / 4850 (2048-point
// chunks order alike): launches that fill the device count for more than groups
// that stay in L2, and past four branches or 256 MB there is nothing left to fill.
constexpr int kXcDefaultBranches = 4;

struct XcWork {
  XcChunks ch;
  int nbr = kXcDefaultBranches; // branches in use, 1..kXcBranches
  XcBranch br[kXcBranches];
  DevBuf Vacc;                  // V accumulators (nao x nao), one or more per branch
  DevBuf ered;                  // energy partials per chunk and block
  // the evaluation's device work as a CUDA graph, captured on the second call
  // with the same arguments and replayed while they stay the same
  cudaGraphExec_t exec = nullptr;
  cudaStream_t cap = nullptr;   // private stream the work is captured on (capture only
                                // records; the graph is launched on the caller's stream)
  const void* g_args[4] = {nullptr, nullptr, nullptr, nullptr};   // P, Vxc, pts, w
  int64_t graph_kernels = 0;    // this library's kernels in the graph
  int calls = 0;
  bool graph_off = false;       // capture failed once: run the launches directly
  ~XcWork() {
    if (exec) cudaGraphExecDestroy(exec);
    if (cap) cudaStreamDestroy(cap);
  }
};

// The SP2 projection of A (m x m symmetric, m <= kSp2ClusterMax) onto its nocc
// lowest eigenvalues in one launch (sp2.cu): X, and rec = {steps, Tr X, 1 when
// converged}; Xg: sp2_cluster_bytes(m) of scratch. kSp2ClusterMax: a copy of X
// fits in a CTA's shared memory.
constexpr int kSp2ClusterMax = 160;
constexpr int kSp2Extra = 2;   // steps after the stopping rule holds: X^2, then 2X - X^2
size_t sp2_cluster_bytes(int m);
void launch_sp2_cluster(const double* A, int m, int nocc, int max_steps, double* Xg, double* X,
                        double* rec, cudaStream_t s);

// Uploads the grid sorted along a Morton curve over 1-Bohr cells, points of a cell
// in their own order (points.cu): pts [n][3] and w [n] on the device, and the
// bounding box {low x, y, z, high x, y, z} of every kXcBox sorted points. pts_host
// and w_host are host arrays. Host synchronizing.
constexpr int kXcBox = 256;
void sort_points(const double* pts_host, const double* w_host, int64_t n, DevBuf& pts, DevBuf& w,
                 std::vector<double>& boxes, cudaStream_t s);
// Cuts n sorted points into chunks of G points, a multiple of kXcBox, and keeps for each chunk the
// shells whose value-and-gradient bound over the chunk's bounding box exceeds
// thresh (uploads the shell lists); forgets any captured graph of ws.
void xc_chunk(const Shells& sh, const int (&nout)[8], int64_t n, const std::vector<double>& boxes,
              int64_t G, double thresh, XcWork& ws);

struct XcParams {
  double x_scale = 0.75;        // PBE exchange share (PBE0)
  double c_scale = 1.0;         // PBE correlation share
  double rho_thresh = 1e-10;    // points at or below this density are left out
};

// E_xc of the closed-shell density P (nao x nao, symmetric, device) and, when
// Vxc != nullptr, its P-gradient symmetrized (device, nao x nao), over the grid
// points pts [n][3] with weights w [n] (device, in sort_points' order), chunk
// by chunk as ws.ch lays them out, on the context's branch streams forked from
// and joined to s. Returns E_xc (host synchronizing); Vcopy, when given,
// receives a copy of Vxc before that.
double xc_energy_fock(const Context& c, const OrbView& ov, const double* pts, const double* w,
                      const double* P, double* Vxc, const XcParams& xp, XcWork& ws,
                      cudaStream_t s, double* Vcopy = nullptr);

// Becke cell weights: w[i] = raw[i] * P_owner(i) / sum_A P_A at point i
void launch_becke_partition(const double* pts, const int* owner, const double* raw, int64_t n,
                            const double* atom_xyz, const double* bragg, int natom, double* w,
                            cudaStream_t s);

}  // namespace dfjk
