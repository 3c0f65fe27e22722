// Surface reconstruction for getIsomesh(): the marker particles' implicit
// surface, polygonised by marching cubes on a grid subdivided `s` times,
// then smoothed.  This restates, on the GPU, what the reference's mesher
// thread does at the first substep of every frame
// (FluidSimulation::_outputSurfaceMeshThread, fluidsimulation.cpp:5150-5219):
//
//   ParticleMesher::meshParticles (particlemesher.cpp:35-55) with one compute
//   chunk: the 10-node blocks that hold particles, feathered by one block
//   (:116-137); the chunk around them (:139-282); per node the smallest
//   |node - p| - r over the particles whose search box covers it, in the
//   frame of the node's block (:406-549, :618-664), negated (:472-478);
//   ScalarField's clamp of solid nodes to the surface threshold
//   (scalarfield.cpp:372-448); Polygonizer3d (polygonizer3d.cpp:380-675):
//   cells with nodes on both sides, vertices on cut edges placed by linear
//   interpolation and kept out of the solid (:455-491), numbered in the order
//   the reference's scan over cells and edges creates them; triangles from
//   the marching-cubes table; the chunk offset and the scale/unscale of
//   meshParticles; TriangleMesh::smooth (trianglemesh.cpp:481-585).
//
// The GPU work is organised for parallelism, not as the reference's loops:
//   * field: of most nodes only the side is needed (is a particle within r,
//     is the node in the solid), as a bit; the value only at the ends of the
//     cut edges.  Both come from a search for the node's nearest particle
//     through the cell bins (sqrt and the subtraction of r are monotone, so
//     min(|d|) - r comes out exactly);
//   * numbering: a vertex belongs to the first cell in flat order that holds
//     its edge (for an edge, the cell below it in every perpendicular axis
//     where there is one).  So a cell's new vertices and its triangles are
//     counted from its cube index and position alone; a scan over cells
//     gives every cell its first vertex and triangle, and the vertex of any
//     edge is found from the cell that creates it.  The numbering is the
//     reference's, with no sequential pass;
//   * smoothing: vertex -> triangle lists by counting sort, each list sorted
//     by triangle index so the neighbour sums add in the reference's order.
// Arithmetic follows the reference operation by operation (the library is
// built with --fmad=false): float distances, FP64 interpolation fractions
// and solid-level-set samples, float vertex arithmetic.  Vertices and
// triangles come out identical to the reference's for the same particles.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/flip3d.h"
#include "flip_device.cuh"

namespace flip {
namespace {

constexpr int MB = 10;          // ParticleMesher::_blockwidth (particlemesher.h:190)
constexpr int MESH_TPB = 256;
constexpr int SEARCH_TPB = 128;   // searches differ in length: small CTAs
constexpr int CELLS_PER_THREAD = 8;
constexpr int TILE = MESH_TPB * CELLS_PER_THREAD;   // cells per scan tile

// The marching-cubes triangle table (Lorensen and Cline's cases as Paul
// Bourke published them, the table the reference's Polygonizer3d uses,
// polygonizer3d.cpp:97-354), re-encoded: case q's triangles are the edge ids
// in the 4-bit fields of kTri[q], lowest first, three per triangle, ended by
// 0xF.  The edge table is not stored: edge e is cut when its two corners
// differ in the cube index.
__device__ const unsigned long long kTri[256] = {
    0xffffffffffffffffull, 0xfffffffffffff380ull, 0xfffffffffffff910ull, 0xffffffffff189381ull,
    0xfffffffffffffa21ull, 0xffffffffffa21380ull, 0xffffffffff920a29ull, 0xfffffff89a8a2382ull,
    0xfffffffffffff2b3ull, 0xffffffffff0b82b0ull, 0xffffffffffb32091ull, 0xfffffffb89b912b1ull,
    0xffffffffff3ab1a3ull, 0xfffffffab8a801a0ull, 0xfffffff9ab9b3093ull, 0xffffffffffb8aa89ull,
    0xfffffffffffff874ull, 0xffffffffff437034ull, 0xffffffffff748910ull, 0xfffffff137174914ull,
    0xffffffffff748a21ull, 0xfffffffa21403743ull, 0xfffffff748209a29ull, 0xffff4973727929a2ull,
    0xffffffffff2b3748ull, 0xfffffff40242b74bull, 0xfffffffb32748109ull, 0xffff1292b9b49b74ull,
    0xfffffff487ab31a3ull, 0xffff4b7401b41ab1ull, 0xffff30bab9b09874ull, 0xfffffffab99b4b74ull,
    0xfffffffffffff459ull, 0xffffffffff380459ull, 0xffffffffff051450ull, 0xfffffff513538458ull,
    0xffffffffff459a21ull, 0xfffffff594a21803ull, 0xfffffff204245a25ull, 0xffff8434535235a2ull,
    0xffffffffffb32459ull, 0xfffffff594b802b0ull, 0xfffffffb32510450ull, 0xffff584b82852512ull,
    0xfffffff45931ab3aull, 0xffffab81a8180594ull, 0xffff30bab5b05045ull, 0xfffffffb8aa85845ull,
    0xffffffffff975879ull, 0xfffffff375359039ull, 0xfffffff751710870ull, 0xffffffffff753351ull,
    0xfffffff21a759879ull, 0xffff37503505921aull, 0xffff25a758528208ull, 0xfffffff7533525a2ull,
    0xfffffff2b3987597ull, 0xffffb72029279759ull, 0xffff751871810b32ull, 0xfffffff51771b12bull,
    0xffffb3a31a758859ull, 0xf0aba010b7905075ull, 0xf07570805a30b0abull, 0xffffffffff5b75abull,
    0xfffffffffffff56aull, 0xffffffffff6a5380ull, 0xffffffffff6a5109ull, 0xfffffff6a5891381ull,
    0xffffffffff162561ull, 0xfffffff803621561ull, 0xfffffff620609569ull, 0xffff823625285895ull,
    0xffffffffff56ab32ull, 0xfffffff56a02b80bull, 0xfffffff6a5b32910ull, 0xffffb892b92916a5ull,
    0xfffffff315356b36ull, 0xffff6b51505b0b80ull, 0xffff9505606306b3ull, 0xfffffff89bb96956ull,
    0xffffffffff8746a5ull, 0xfffffffa56374034ull, 0xfffffff7486a5091ull, 0xffff49737179156aull,
    0xfffffff874156216ull, 0xffff743403625521ull, 0xffff620560509748ull, 0xf962695923497937ull,
    0xfffffff56a4872b3ull, 0xffffb720242746a5ull, 0xffff6a5b32874910ull, 0xf6a54b7b492b9129ull,
    0xffff6b51535b3748ull, 0xfb404b7b016b5b15ull, 0xf74836b630560950ull, 0xffff9b7974b96956ull,
    0xffffffffffa4694aull, 0xfffffff380a946a4ull, 0xfffffff04606a10aull, 0xffffa16468618138ull,
    0xfffffff462421941ull, 0xffff462942921803ull, 0xffffffffff624420ull, 0xfffffff624428238ull,
    0xfffffff32b46a94aull, 0xffff6a4a94b82280ull, 0xffffa164606102b3ull, 0xf1b8b12184a16146ull,
    0xffff36b319639469ull, 0xf14641916b0181b8ull, 0xfffffff4600636b3ull, 0xffffffffff86b846ull,
    0xfffffffa98a876a7ull, 0xffffa76a907a0370ull, 0xffff0818717a176aull, 0xfffffff37117a76aull,
    0xffff768981861621ull, 0xf937390976192962ull, 0xfffffff206607087ull, 0xffffffffff276237ull,
    0xffff76898a86ab32ull, 0xf7a9a76790b72702ull, 0xfb32a767a1871081ull, 0xffff17616a71b12bull,
    0xf63136b619768698ull, 0xffffffffff76b190ull, 0xffff06b0b3607087ull, 0xfffffffffffff6b7ull,
    0xfffffffffffffb67ull, 0xffffffffff67b803ull, 0xffffffffff67b910ull, 0xfffffff67b138918ull,
    0xffffffffff7b621aull, 0xfffffff7b6803a21ull, 0xfffffff7b69a2092ull, 0xffff89a38a3a27b6ull,
    0xffffffffff726327ull, 0xfffffff026067807ull, 0xfffffff910732672ull, 0xffff678891681261ull,
    0xfffffff73171a67aull, 0xffff801781a7167aull, 0xffff7a69a0a70730ull, 0xfffffff9a88a7a67ull,
    0xffffffffff68b486ull, 0xfffffff640603b63ull, 0xfffffff109648b68ull, 0xffff63b139369649ull,
    0xfffffff1a28b6486ull, 0xffff640b60b03a21ull, 0xffff9a2920b648b4ull, 0xf36463b34923a39aull,
    0xfffffff264248328ull, 0xffffffffff264240ull, 0xffff834642432091ull, 0xfffffff642241491ull,
    0xffff1a6648168318ull, 0xfffffff40660a01aull, 0xf39a9303a6834364ull, 0xffffffffff4a649aull,
    0xffffffffffb67594ull, 0xfffffff67b594380ull, 0xfffffffb67045105ull, 0xffff51345343867bull,
    0xfffffffb6721a459ull, 0xffff594380a217b6ull, 0xffff204a24a45b67ull, 0xf67b25a523453843ull,
    0xfffffff945267327ull, 0xffff786260680459ull, 0xffff045051673263ull, 0xf851584812786826ull,
    0xffff73167161a459ull, 0xf459078701671a61ull, 0xfa737a6a305a4a04ull, 0xffffa84a458a7a67ull,
    0xfffffff98b9b6596ull, 0xffff590650360b63ull, 0xffffb65510b508b0ull, 0xfffffff1355363b6ull,
    0xffff65b8b9b59a21ull, 0xfa21965690b603b0ull, 0xf52025a50865b58bull, 0xffff35a3a25363b6ull,
    0xffff283265825985ull, 0xfffffff260069659ull, 0xf826283865081851ull, 0xffffffffff612651ull,
    0xf698965683a61631ull, 0xffff06505960a01aull, 0xffffffffffa65830ull, 0xfffffffffffff65aull,
    0xffffffffffb57a5bull, 0xfffffff03857ba5bull, 0xfffffff091ba57b5ull, 0xffff1381897ba57aull,
    0xfffffff15717b21bull, 0xffffb27571721380ull, 0xffff7b2209729579ull, 0xf289823295b27257ull,
    0xfffffff573532a52ull, 0xffff52a578258028ull, 0xffff2a37353a5109ull, 0xf25752a278129289ull,
    0xffffffffff573531ull, 0xfffffff571170780ull, 0xfffffff735539309ull, 0xffffffffff795789ull,
    0xfffffff8ba8a5485ull, 0xffff03bba50b5405ull, 0xffff54aba8a48910ull, 0xf41314943b54a4baull,
    0xffff8548b2582152ull, 0xfb151b2b543b0b40ull, 0xf58b8545b2950520ull, 0xffffffffff3b2549ull,
    0xffff483543253a52ull, 0xfffffff0244252a5ull, 0xf910854583a532a3ull, 0xffff2492914252a5ull,
    0xfffffff153358548ull, 0xffffffffff501540ull, 0xffff530509358548ull, 0xfffffffffffff549ull,
    0xfffffffba9b947b4ull, 0xffffba97b9794380ull, 0xffffb470414b1ba1ull, 0xf4bab474a1843413ull,
    0xffff219b294b97b4ull, 0xf3801b2b197b9479ull, 0xfffffff04224b47bull, 0xffff42343824b47bull,
    0xffff947732972a92ull, 0xf70207872a4797a9ull, 0xfa040a1a472a3a73ull, 0xffffffffff4782a1ull,
    0xfffffff317714194ull, 0xffff178180714194ull, 0xffffffffff347304ull, 0xfffffffffffff784ull,
    0xffffffffff8ba8a9ull, 0xfffffffa9bb93903ull, 0xfffffffba88a0a10ull, 0xffffffffffa3ba13ull,
    0xfffffff8b99b1b21ull, 0xffff9b2921b93903ull, 0xffffffffffb08b20ull, 0xfffffffffffffb23ull,
    0xfffffff98aa82832ull, 0xffffffffff2902a9ull, 0xffff8a1810a82832ull, 0xfffffffffffff2a1ull,
    0xffffffffff819831ull, 0xfffffffffffff190ull, 0xfffffffffffff830ull, 0xffffffffffffffffull,
};

// Cube corners (Grid3d::getGridIndexVertices, grid3d.h:304-313): corner q at
// (i + kCx[q], j + kCy[q], k + kCz[q]).
#define FLIP_CORNERS_X {0, 1, 1, 0, 0, 1, 1, 0}
#define FLIP_CORNERS_Y {0, 0, 0, 0, 1, 1, 1, 1}
#define FLIP_CORNERS_Z {0, 0, 1, 1, 0, 0, 1, 1}
__constant__ int kCx[8] = FLIP_CORNERS_X;
__constant__ int kCy[8] = FLIP_CORNERS_Y;
__constant__ int kCz[8] = FLIP_CORNERS_Z;
// Edges in the reference's order (polygonizer3d.cpp:495-630): the corners
// interpolated from and to, the axis of the edge and the corner it starts
// from along that axis (which names the edge in the grid of edges).
#define FLIP_EDGE_DIR {0, 2, 0, 2, 0, 2, 0, 2, 1, 1, 1, 1}
#define FLIP_EDGE_ORG {0, 1, 3, 0, 4, 5, 7, 4, 0, 1, 2, 3}
__constant__ int kEa[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3};
__constant__ int kEb[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
__constant__ int kEdir[12] = FLIP_EDGE_DIR;
__constant__ int kEorg[12] = FLIP_EDGE_ORG;

// Edges whose two corners differ in the cube index: edges 0-3 join corner e of
// the lower four with the next one round, 4-7 of the upper four, 8-11 a lower
// corner with the one above.
__device__ __forceinline__ unsigned cut_mask(int q) {
    const unsigned lo = q & 15, hi = (unsigned)q >> 4;
    return (lo ^ (lo >> 1 | (lo & 1) << 3)) | (hi ^ (hi >> 1 | (hi & 1) << 3)) << 4 | (lo ^ hi) << 8;
}
// A case's fields past its last triangle are all 0xF, and an edge id is below 12.
__device__ __forceinline__ int tri_count(int q) { return (16 - __clzll(~(long long)kTri[q]) / 4) / 3; }
// Edges that lie along an axis or start from its upper corner.
__host__ __device__ constexpr unsigned edges_off(int axis) {
    constexpr int c[3][8] = {FLIP_CORNERS_X, FLIP_CORNERS_Y, FLIP_CORNERS_Z}, dir[12] = FLIP_EDGE_DIR, org[12] = FLIP_EDGE_ORG;
    unsigned m = 0;
    for (int e = 0; e < 12; e++)
        if (dir[e] == axis || c[axis][org[e]] == 1) m |= 1u << e;
    return m;
}
// Edges that cell (i, j, k) creates: the first cell in flat order holding an
// edge is the one below it in each perpendicular axis, where that cell exists.
__device__ __forceinline__ unsigned created_mask(int i, int j, int k) {
    constexpr unsigned x = edges_off(0), y = edges_off(1), z = edges_off(2);
    return (i == 0 ? 0xfffu : x) & (j == 0 ? 0xfffu : y) & (k == 0 ? 0xfffu : z);
}

// Nodal solid level set at a point, in FP64 as Interpolation::
// trilinearInterpolate(vec3, dx, grid) evaluates it (interpolation.cpp:61-113):
// the cell by floor(p / dx), the offset from the cell's float corner, the
// eight weights; nodes outside the grid count as 0.
__device__ double solid_sample(const MeshFrame &m, const float *S, float px, float py, float pz) {
    const int i = (int)floor((double)px * m.invdx), j = (int)floor((double)py * m.invdx),
              k = (int)floor((double)pz * m.invdx);
    const float gx = (float)((double)(float)i * m.dx), gy = (float)((double)(float)j * m.dx),
                gz = (float)((double)(float)k * m.dx);
    const double x = (double)__fsub_rn(px, gx) * m.invdx, y = (double)__fsub_rn(py, gy) * m.invdx,
                 z = (double)__fsub_rn(pz, gz) * m.invdx;
    const int ni = m.I + 1, nj = m.J + 1, nk = m.K + 1;
    auto at = [&](int a, int b, int c) -> double {
        return (a >= 0 && b >= 0 && c >= 0 && a < ni && b < nj && c < nk)
                   ? (double)S[(long long)a + (long long)ni * ((long long)b + (long long)nj * c)]
                   : 0.0;
    };
    const double p0 = at(i, j, k), p1 = at(i + 1, j, k), p2 = at(i, j + 1, k), p3 = at(i, j, k + 1),
                 p4 = at(i + 1, j, k + 1), p5 = at(i, j + 1, k + 1), p6 = at(i + 1, j + 1, k),
                 p7 = at(i + 1, j + 1, k + 1);
    return p0 * (1 - x) * (1 - y) * (1 - z) + p1 * x * (1 - y) * (1 - z) + p2 * (1 - x) * y * (1 - z) +
           p3 * (1 - x) * (1 - y) * z + p4 * x * (1 - y) * z + p5 * (1 - x) * y * z + p6 * x * y * (1 - z) +
           p7 * x * y * z;
}

// The sign of solid_sample where it is plain, else 0: all nodes around the point
// of one sign and within a factor of 20, far beyond what the rounding of the
// weights (which add up to 1, none below -1e-3) can turn, or a value
// interpolated in 32 bits of more than 1% of the largest of them.  The cell is
// found in 32 bits, and where the point is within 0.01 of a cell's face, the
// nodes of both cells count.  Spares nearly all of the FP64 interpolation: an
// SM does two FP64 operations a cycle.
__device__ __forceinline__ int solid_sign(const MeshFrame &m, const float *S, float px, float py, float pz) {
    const float gx = px * m.invdxf, gy = py * m.invdxf, gz = pz * m.invdxf;
    const int i0 = (int)floorf(gx - 0.01f), i1 = (int)floorf(gx + 0.01f) + 1, j0 = (int)floorf(gy - 0.01f),
              j1 = (int)floorf(gy + 0.01f) + 1, k0 = (int)floorf(gz - 0.01f), k1 = (int)floorf(gz + 0.01f) + 1;
    if (i0 < 0 || j0 < 0 || k0 < 0 || i1 > m.I || j1 > m.J || k1 > m.K) return 0;
    const int ni = m.I + 1, nj = m.J + 1;
    float lo = __uint_as_float(0x7f800000u), hi = -lo;
    for (int k = k0; k <= k1; k++)
        for (int j = j0; j <= j1; j++) {
            const float *s = S + i0 + (long long)ni * (j + (long long)nj * k);
            const float a = s[0], b = s[1], c = s[i1 - i0];
            lo = fminf(fminf(lo, a), fminf(b, c));
            hi = fmaxf(fmaxf(hi, a), fmaxf(b, c));
        }
    if (lo > fmaxf(0.05f * hi, 1e-20f)) return 1;
    if (hi < fminf(0.05f * lo, -1e-20f)) return -1;
    // mixed: by interpolation in 32 bits, where it is far from 0
    const int i = min(max((int)floorf(gx), 0), m.I - 1), j = min(max((int)floorf(gy), 0), m.J - 1),
              k = min(max((int)floorf(gz), 0), m.K - 1);
    const float x = gx - (float)i, y = gy - (float)j, z = gz - (float)k;
    const float *s = S + i + (long long)ni * (j + (long long)nj * k);
    auto along = [&](const float *r) { return r[0] + x * (r[1] - r[0]); };
    const float c0 = along(s), c1 = along(s + ni), c2 = along(s + (long long)ni * nj), c3 = along(s + (long long)ni * (nj + 1));
    const float b0 = c0 + y * (c1 - c0), b1 = c2 + y * (c3 - c2), d = b0 + z * (b1 - b0);
    const float sure = fmaxf(0.01f * fmaxf(hi, -lo), 1e-20f);
    return d > sure ? 1 : (d < -sure ? -1 : 0);
}

// Is chunk node (a, b, c) a solid vertex (ScalarField::setSolidSDF,
// scalarfield.cpp:372-395, MeshLevelSet::_trilinearInterpolateSolidGridPointsThread,
// meshlevelset.cpp:309-340)?
// -1: solid, 1: not, 0: the level set has to be interpolated there.
__device__ __forceinline__ int solid_vertex_sign(const MeshFrame &m, const float *S, int a, int b, int c) {
    if (m.solidMode == 2)   // the scalar field's grid is the level set's
        return S[(long long)a + (long long)(m.I + 1) * ((long long)b + (long long)(m.J + 1) * c)] < 0.0f ? -1 : 1;
    if (m.solidMode == 1 && !(a & 1) && !(b & 1) && !(c & 1))   // subdivision 2 at offset 0: even nodes
        return S[(long long)(a >> 1) + (long long)(m.I + 1) * ((long long)(b >> 1) + (long long)(m.J + 1) * (c >> 1))] < 0.0f
                   ? -1
                   : 1;
    return solid_sign(m, S, (float)a * m.subdxf + m.offx, (float)b * m.subdxf + m.offy, (float)c * m.subdxf + m.offz);
}
__device__ bool solid_vertex_value(const MeshFrame &m, const float *S, int a, int b, int c) {
    const float px = __fadd_rn((float)((double)(float)a * m.subdx), m.offx);
    const float py = __fadd_rn((float)((double)(float)b * m.subdx), m.offy);
    const float pz = __fadd_rn((float)((double)(float)c * m.subdx), m.offz);
    const double d = solid_sample(m, S, px, py, pz);
    return m.solidMode == 1 ? (float)d < 0.0f : d < 0.0;
}

// ---------------------------------------------------------------- occupancy
// Blocks holding a particle (ParticleMesher::
// _initializeComputeChunkDataActiveBlocks, particlemesher.cpp:116-137).
__global__ void k_mesh_occupancy(ParticleSoA p, int n, MeshFrame m, uint8_t *occ) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    int at = -1;
    if (t < n) {
        const int bi = exact_floor(p.px[t], m.invBlock, m.invBlockf), bj = exact_floor(p.py[t], m.invBlock, m.invBlockf),
                  bk = exact_floor(p.pz[t], m.invBlock, m.invBlockf);
        if (bi >= 0 && bj >= 0 && bk >= 0 && bi < m.nbI && bj < m.nbJ && bk < m.nbK) at = bi + m.nbI * (bj + m.nbJ * bk);
    }
    // the lane before mostly has the same block to mark
    const int before = __shfl_up_sync(0xffffffffu, at, 1);
    if (at >= 0 && ((threadIdx.x & 31) == 0 || at != before)) occ[at] = 1;
}

// -------------------------------------------------------------- scalar field
// Does the reference's scatter take particle p to node (a, b, c) of block
// (bx, by, bz)?  The count pass's block lists (particlemesher.cpp:400-446) and
// the particle's node box in the block's frame; cx..cz: p in the chunk's frame,
// lx..lz: in the block's.
__device__ __noinline__ bool field_reaches(const MeshFrame &m, float cx, float cy, float cz, float lx, float ly, float lz,
                                           int bx, int by, int bz, int a, int b, int c) {
    const float sr = m.sr;
    const int oi = exact_floor(cx, m.invBlockF, m.invBlockFf), oj = exact_floor(cy, m.invBlockF, m.invBlockFf),
              ok = exact_floor(cz, m.invBlockF, m.invBlockFf);
    const float bpx = (float)((double)(float)oi * (double)m.blockdxF), bpy = (float)((double)(float)oj * (double)m.blockdxF),
                bpz = (float)((double)(float)ok * (double)m.blockdxF);
    bool mine;
    if (__fsub_rn(cx, sr) > bpx && __fsub_rn(cy, sr) > bpy && __fsub_rn(cz, sr) > bpz &&
        __fadd_rn(cx, sr) < __fadd_rn(bpx, m.blockdxF) && __fadd_rn(cy, sr) < __fadd_rn(bpy, m.blockdxF) &&
        __fadd_rn(cz, sr) < __fadd_rn(bpz, m.blockdxF)) {
        mine = oi == bx && oj == by && ok == bz;
    } else {
        mine = bx >= exact_floor(__fsub_rn(cx, sr), m.invBlockF, m.invBlockFf) &&
               bx <= exact_floor(__fadd_rn(cx, sr), m.invBlockF, m.invBlockFf) &&
               by >= exact_floor(__fsub_rn(cy, sr), m.invBlockF, m.invBlockFf) &&
               by <= exact_floor(__fadd_rn(cy, sr), m.invBlockF, m.invBlockFf) &&
               bz >= exact_floor(__fsub_rn(cz, sr), m.invBlockF, m.invBlockFf) &&
               bz <= exact_floor(__fadd_rn(cz, sr), m.invBlockF, m.invBlockFf);
    }
    return mine && a >= exact_floor(__fsub_rn(lx, sr), m.invsub, m.invsubf) &&
           a <= exact_floor(__fadd_rn(lx, sr), m.invsub, m.invsubf) + 1 &&
           b >= exact_floor(__fsub_rn(ly, sr), m.invsub, m.invsubf) &&
           b <= exact_floor(__fadd_rn(ly, sr), m.invsub, m.invsubf) + 1 &&
           c >= exact_floor(__fsub_rn(lz, sr), m.invsub, m.invsubf) &&
           c <= exact_floor(__fadd_rn(lz, sr), m.invsub, m.invsubf) + 1;
}

// The reference scatters every particle over the nodes of its search box
// (hundreds of them); a node's value is that of its nearest particle, since the
// rounded square root and the subtraction of r are monotone.  So a node looks
// for it.  A Seeker holds what a search needs of its node and tests particles.
template <bool SIGN>
struct Seeker {
    const ParticleSoA &p;
    const MeshFrame &m;
    int A, B, C;
    float bofx, bofy, bofz, nx, ny, nz;   // the frame of the node's block, the node there
    float px, py, pz;                     // the node in the simulation's frame
    float best;                           // SIGN: best < 0 once one nearer than r is found
    __device__ Seeker(const ParticleSoA &p_, const MeshFrame &m_, int A_, int B_, int C_)
        : p(p_), m(m_), A(A_), B(B_), C(C_) {
        const int bx = A / MB, by = B / MB, bz = C / MB;
        bofx = m.blockPos[0][bx];
        bofy = m.blockPos[1][by];
        bofz = m.blockPos[2][bz];
        nx = m.nodePos[A - bx * MB];
        ny = m.nodePos[B - by * MB];
        nz = m.nodePos[C - bz * MB];
        px = m.offx + (float)A * m.subdxf;
        py = m.offy + (float)B * m.subdxf;
        pz = m.offz + (float)C * m.subdxf;
        best = SIGN ? m.signReach * m.signReach : __uint_as_float(0x7f800000u);
    }
    // squared distance in the frame of the node's block, as the reference finds
    // it (_scalarFieldProducerThread, particlemesher.cpp:498-549)
    __device__ float dist2(float qx, float qy, float qz) const {
        const float dx = __fsub_rn(nx, __fsub_rn(__fsub_rn(qx, m.offx), bofx)),
                    dy = __fsub_rn(ny, __fsub_rn(__fsub_rn(qy, m.offy), bofy)),
                    dz = __fsub_rn(nz, __fsub_rn(__fsub_rn(qz, m.offz), bofz));
        return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    }
    // the chunk's box, expanded (particlemesher.cpp:287-301, aabb.cpp:122-133)
    __device__ bool in_box(float qx, float qy, float qz) const {
        return qx >= m.bbx && qy >= m.bby && qz >= m.bbz && qx < m.bhx && qy < m.bhy && qz < m.bhz;
    }
    __device__ void test(float qx, float qy, float qz) {
        const float d2 = dist2(qx, qy, qz);
        if (!(d2 < best) || (SIGN && !(__fsqrt_rn(d2) < m.r)) || !in_box(qx, qy, qz)) return;
        if (!(d2 < m.near2)) {
            const float cx = __fsub_rn(qx, m.offx), cy = __fsub_rn(qy, m.offy), cz = __fsub_rn(qz, m.offz);
            const int bx = A / MB, by = B / MB, bz = C / MB;
            if (!field_reaches(m, cx, cy, cz, __fsub_rn(cx, bofx), __fsub_rn(cy, bofy), __fsub_rn(cz, bofz), bx, by, bz,
                               A - bx * MB, B - by * MB, C - bz * MB))
                return;
        }
        best = SIGN ? -1.0f : d2;
    }
    __device__ void look(int from, int to, int step) {   // particles from, from + step, ...
        for (int t = from; t < to; t += 4 * step) {
            float qx[4], qy[4], qz[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {   // four at a time, so that their loads overlap
                const int tq = t + q * step < to ? t + q * step : t;
                qx[q] = p.px[tq];
                qy[q] = p.py[tq];
                qz[q] = p.pz[tq];
            }
            // a first look in plain coordinates; `slack` is far above what
            // their rounding and the block frame's make of a squared distance
            bool hit = false;
            const float bar = best + m.slack;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float ex = qx[q] - px, ey = qy[q] - py, ez = qz[q] - pz;
                hit |= __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, ex * ex)) < bar;
            }
            if (!hit) continue;
            // the nearest of the four; below near2 its list and box surely hold
            // the node, which leaves nothing to look up
            float d2 = dist2(qx[0], qy[0], qz[0]), x = qx[0], y = qy[0], z = qz[0];
#pragma unroll
            for (int q = 1; q < 4; q++) {
                const float e2 = dist2(qx[q], qy[q], qz[q]);
                const bool nearer = e2 < d2;
                d2 = nearer ? e2 : d2;
                x = nearer ? qx[q] : x;
                y = nearer ? qy[q] : y;
                z = nearer ? qz[q] : z;
            }
            if (!(d2 < best)) continue;
            if (d2 < m.near2 && in_box(x, y, z)) {
                if (!SIGN) best = d2;
                else if (__fsqrt_rn(d2) < m.r) best = -1.0f;
            } else {
                for (int q = 0; q < 4; q++)
                    if (t + q * step < to) test(p.px[t + q * step], p.py[t + q * step], p.pz[t + q * step]);
            }
            if (SIGN && best < 0.0f) return;
        }
    }
};

// A search by GROUP lanes (all of a group call it with the same node): its own
// cell together, then the rows of cells around it, nearest first, a row a lane,
// as long as one can hold a nearer particle.  Returns the squared distance to
// the nearest particle, +inf without one; with SIGN 0 if one is nearer than r,
// else +inf.  Particles beyond near2 have to be looked up in the lists, with
// FP64: a first pass leaves them out, and mostly finds a nearer one.
template <bool SIGN, int GROUP>
__device__ float nearest(const ParticleSoA &p, const int *cellStart, const MeshFrame &m, int A, int B, int C) {
    const float kInf = __uint_as_float(0x7f800000u);
    const int lane = threadIdx.x & 31, g = lane & (GROUP - 1);
    const unsigned group = ((1u << GROUP) - 1) << (lane - g);
    Seeker<SIGN> sk(p, m, A, B, C);
    // the cell the node lies in and its place there, in cells
    const float gx = m.cellAt(m.offx, A), gy = m.cellAt(m.offy, B), gz = m.cellAt(m.offz, C);
    const int i = (int)floorf(gx), j = (int)floorf(gy), k = (int)floorf(gz);
    const float fy = gy - (float)j, fz = gz - (float)k;
    auto least = [&]() {
#pragma unroll
        for (int o = GROUP / 2; o > 0; o >>= 1) sk.best = fminf(sk.best, __shfl_xor_sync(group, sk.best, o));
    };
    // squared distance along an axis to the cells o away, less a margin far
    // above the rounding of the positions
    auto away = [&](int o, float f) {
        const float d = fmaxf((o > 0 ? (float)o - f : (o < 0 ? f - (float)(o + 1) : 0.0f)) - 0.01f, 0.0f) * m.dxf;
        return d * d;
    };
    const int sy = fy < 0.5f ? -1 : 1, sz = fz < 0.5f ? -1 : 1;   // towards the nearer side
    const float all = sk.best;
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        const float bound = pass == 0 ? fminf(all, m.near2) : all;
        sk.best = bound;
        if (i < m.I && j < m.J && k < m.K) {
            const long long own = i + (long long)m.I * (j + (long long)m.J * k);
            sk.look(cellStart[own] + g, cellStart[own + 1], GROUP);
        }
        __syncwarp(group);
        least();
#pragma unroll 1
        for (int n0 = 0; n0 < m.nrows && m.rows[n0].least < sk.best; n0 += GROUP) {
            if (n0 + g < m.nrows) {
                const MeshRow row = m.rows[n0 + g];
                const int oy = sy * row.y, oz = sz * row.z, y = j + oy, z = k + oz;
                const float d = away(oy, fy) + away(oz, fz);
                if (d < sk.best && y >= 0 && z >= 0 && y < m.J && z < m.K) {
                    // how far along the row a nearer particle can be
                    const float w = fminf(sqrtf(sk.best - d), m.reach) * m.invdxf + 0.02f;
                    const int x0 = max((int)floorf(gx - w), 0), x1 = min((int)floorf(gx + w), m.I - 1);
                    const long long base = (long long)m.I * (y + (long long)m.J * z);
                    if (x0 <= x1) sk.look(cellStart[base + x0], cellStart[base + x1 + 1], 1);
                }
            }
            __syncwarp(group);
            least();
        }
        if (sk.best < bound) return SIGN ? 0.0f : sk.best;
        if (bound == all) break;
    }
    return kInf;
}
__device__ __forceinline__ bool block_active(const MeshFrame &m, const uint8_t *active, int A, int B, int C) {
    return active[A / MB + m.cbI * (B / MB + m.cbJ * (C / MB))];
}

// Cells with a particle as bits, 32 along x to a word (a warp a word), and the
// cells with one within R cells of them along each axis: nodes elsewhere are
// outside without a search, most of the air.
__global__ void __launch_bounds__(MESH_TPB) k_mesh_occupied(const int *cellStart, MeshFrame m, unsigned *occupied) {
    const long long word = (long long)blockIdx.x * (MESH_TPB / 32) + (threadIdx.x >> 5);
    if (word >= (long long)m.wpc * m.J * m.K) return;
    int wx, j, k;
    unflatten(word, m.wpc, m.J, wx, j, k);
    const int i = wx * 32 + (threadIdx.x & 31);
    const int *s = cellStart + i + (long long)m.I * (j + (long long)m.J * k);
    const unsigned w = __ballot_sync(0xffffffffu, i < m.I && s[0] != s[1]);
    if ((threadIdx.x & 31) == 0) occupied[word] = w;
}
__global__ void __launch_bounds__(MESH_TPB) k_mesh_around(MeshFrame m, const unsigned *occupied, int R, unsigned *around) {
    const long long word = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (word >= (long long)m.wpc * m.J * m.K) return;
    int wx, j, k;
    unflatten(word, m.wpc, m.J, wx, j, k);
    unsigned w = 0, below = 0, above = 0;   // the rows' words together
    for (int z = max(k - R, 0); z <= min(k + R, m.K - 1); z++)
        for (int y = max(j - R, 0); y <= min(j + R, m.J - 1); y++) {
            const unsigned *row = occupied + (long long)m.wpc * (y + (long long)m.J * z);
            w |= row[wx];
            if (wx > 0) below |= row[wx - 1];
            if (wx + 1 < m.wpc) above |= row[wx + 1];
        }
    unsigned out = w;
    for (int q = 1; q <= R; q++) out |= __funnelshift_l(below, w, q) | __funnelshift_r(w, above, q);
    around[word] = out;
}

__device__ __forceinline__ bool near_particles(const MeshFrame &m, const unsigned *around, int A, int B, int C) {
    if (!around) return true;
    const int i = min((int)m.cellAt(m.offx, A), m.I - 1), j = min((int)m.cellAt(m.offy, B), m.J - 1),
              k = min((int)m.cellAt(m.offz, C), m.K - 1);
    return around[(i >> 5) + (long long)m.wpc * (j + (long long)m.J * k)] >> (i & 31) & 1u;
}

// Which nodes are inside (field above the threshold, not solid), as bits, 32
// along x to a word: all that the polygoniser asks of a node, but for those at
// the ends of a cut edge.  A warp a word.  A lane looks at its node's own cell,
// which decides nearly all nodes of the liquid; the air is decided without
// particles; the nodes left, near the surface, are searched by groups of lanes.
// Nodes where the solid level set has to be interpolated in FP64, a few at the
// walls' ends of many rows, go to a list (as long as it has room) for
// k_mesh_walls, which works on full warps.
// Bound by the searches near the surface and their latency: 345 us at 128^3,
// subdivision 2 (17M nodes), where scattering every particle over its box took
// 2250 us for all values; 21 us at 71x59x83, subdivision 1.  The searches grow with the
// particles' radius, but less than the boxes did: whole meshes of a 64^3 dam,
// subdivision 2, took 876 us where the scatter took 1462 at marker particle scale 1,
// 345 (943) at 3, 393 (3256) at 8 and 463 (7465) at 12; of 20000 lone particles in
// 128^3 cells 2.2 ms (10.5) at 3 and 8.1 (15.8) at 12.
__global__ void __launch_bounds__(SEARCH_TPB, 1024 / SEARCH_TPB) k_mesh_inside(ParticleSoA p, const int *cellStart, MeshFrame m,
                                                                               const uint8_t *active, const unsigned *around,
                                                                               const float *solidPhi, unsigned *inside,
                                                                               int *walls, int room, int *nwalls) {
    __shared__ int lists[SEARCH_TPB];
    __shared__ unsigned founds[SEARCH_TPB / 32];
    const int lane = threadIdx.x & 31;
    int *list = lists + (threadIdx.x - lane);
    unsigned *found = founds + (threadIdx.x >> 5);
    const long long word = (long long)blockIdx.x * (SEARCH_TPB / 32) + (threadIdx.x >> 5);
    if (word >= (long long)m.wpr * m.nj * m.nk) return;
    int wx, B, C;
    unflatten(word, m.wpr, m.nj, wx, B, C);
    const int A = wx * 32 + lane;
    bool in = false, open = false;
    if (A < m.ni && block_active(m, active, A, B, C) && near_particles(m, around, A, B, C)) {
        Seeker<true> sk(p, m, A, B, C);
        const int i = (int)floorf(m.cellAt(m.offx, A)), j = (int)floorf(m.cellAt(m.offy, B)), k = (int)floorf(m.cellAt(m.offz, C));
        if (i < m.I && j < m.J && k < m.K) {
            const long long own = i + (long long)m.I * (j + (long long)m.J * k);
            sk.look(cellStart[own], cellStart[own + 1], 1);
        }
        in = sk.best < 0.0f;
        open = !in;
    }
    const unsigned opens = __ballot_sync(0xffffffffu, open);
    if (opens) {
        if (open) list[__popc(opens & ((1u << lane) - 1u))] = lane;
        if (lane == 0) *found = 0;
        __syncwarp();
        for (int n = lane / 4; n < __popc(opens); n += 8) {
            const int t = list[n];
            if (nearest<true, 4>(p, cellStart, m, wx * 32 + t, B, C) == 0.0f && lane % 4 == 0) atomicOr(found, 1u << t);
        }
        __syncwarp();
        in |= *found >> lane & 1u;
    }
    int sign = in ? solid_vertex_sign(m, solidPhi, A, B, C) : -1;
    if (sign == 0) {
        const int at = atomicAdd(nwalls, 1);
        if (at < room) walls[at] = (int)(word * 32 + lane);
        else sign = solid_vertex_value(m, solidPhi, A, B, C) ? -1 : 1;
    }
    const unsigned w = __ballot_sync(0xffffffffu, sign > 0);
    if (lane == 0) inside[word] = w;
}
__global__ void __launch_bounds__(MESH_TPB) k_mesh_walls(MeshFrame m, const float *solidPhi, const int *walls, int room,
                                                         const int *nwalls, unsigned *inside) {
    const int n = min(*nwalls, room);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const unsigned t = (unsigned)walls[q];
        int wx, b, c;
        unflatten(t >> 5, m.wpr, m.nj, wx, b, c);
        if (!solid_vertex_value(m, solidPhi, wx * 32 + (int)(t & 31), b, c)) atomicOr(&inside[t >> 5], 1u << (t & 31));
    }
}

// ------------------------------------------------------------------- cells
__device__ __forceinline__ unsigned inside_bit(const MeshFrame &m, const unsigned *inside, int a, int b, int c) {
    return inside[(a >> 5) + (long long)m.wpr * ((long long)b + (long long)m.nj * c)] >> (a & 31) & 1u;
}
// A node's field value: of its nearest particle, 0 in the solid.
template <int GROUP>
__device__ float node_value(const ParticleSoA &p, const int *cellStart, const MeshFrame &m, const uint8_t *active,
                            const unsigned *inside, int a, int b, int c) {
    const float kInf = __uint_as_float(0x7f800000u);
    const float best = block_active(m, active, a, b, c) ? nearest<false, GROUP>(p, cellStart, m, a, b, c) : kInf;
    const float f = -(best == kInf ? m.maxd : fminf(m.maxd, __fsub_rn(__fsqrt_rn(best), m.r)));
    return f > 0.0f && !inside_bit(m, inside, a, b, c) ? 0.0f : f;
}
__device__ __forceinline__ int cube_index(const MeshFrame &m, const unsigned *inside, int i, int j, int k) {
    const unsigned *row = inside + (i >> 5) + (long long)m.wpr * ((long long)j + (long long)m.nj * k);
    const bool across = (i & 31) == 31;
    auto pair = [&](long long o) {   // nodes i and i + 1 of a row
        return across ? row[o] >> 31 | (row[o + 1] & 1u) << 1 : row[o] >> (i & 31) & 3u;
    };
    // corners 0 1 / 3 2 below, 4 5 / 7 6 above (kCx, kCy, kCz)
    const unsigned a = pair(0), b = pair((long long)m.wpr * m.nj), c = pair(m.wpr), d = pair((long long)m.wpr * (m.nj + 1));
    return (int)(a | (b >> 1) << 2 | (b & 1) << 3 | c << 4 | (d >> 1) << 6 | (d & 1) << 7);
}

// inclusive warp scan of int2, then the block's exclusive prefix and total
__device__ int2 block_scan_int2(int2 v, int2 *total) {
    __shared__ int2 wsum[MESH_TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int2 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, x.x, o), b = __shfl_up_sync(0xffffffffu, x.y, o);
        if (lane >= o) { x.x += a; x.y += b; }
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int2 before = make_int2(0, 0), tot = make_int2(0, 0);
    for (int w = 0; w < MESH_TPB / 32; w++) {
        if (w < warp) { before.x += wsum[w].x; before.y += wsum[w].y; }
        tot.x += wsum[w].x;
        tot.y += wsum[w].y;
    }
    __syncthreads();
    *total = tot;
    return make_int2(before.x + x.x - v.x, before.y + x.y - v.y);
}

// Per cell: cube index; per tile: vertices created and triangles (their order
// within a tile does not matter here, so neighbouring threads take
// neighbouring cells).
__global__ void __launch_bounds__(MESH_TPB) k_mesh_count(MeshFrame m, const unsigned *inside, long long ncells,
                                                         uint8_t *cube, int2 *tileSums) {
    const long long base = (long long)blockIdx.x * TILE + threadIdx.x;
    int2 own = make_int2(0, 0);
    const int ci = m.ni - 1, cj = m.nj - 1;
    for (int q = 0; q < CELLS_PER_THREAD; q++) {
        const long long c = base + q * MESH_TPB;
        if (c >= ncells) break;
        int i, j, k;
        unflatten(c, ci, cj, i, j, k);
        const int cq = cube_index(m, inside, i, j, k);
        cube[c] = (uint8_t)cq;
        if (cq != 0 && cq != 255) {
            own.x += __popc(cut_mask(cq) & created_mask(i, j, k));
            own.y += tri_count(cq);
        }
    }
    int2 tot;
    block_scan_int2(own, &tot);
    if (threadIdx.x == 0) tileSums[blockIdx.x] = tot;
}

// Exclusive scan of the tile sums in place (one CTA, any number of tiles);
// the totals to totals[0..1].
__global__ void __launch_bounds__(MESH_TPB) k_mesh_scan_tiles(int2 *tileSums, int ntiles, int *totals) {
    constexpr int PER = 8;
    int2 carry = make_int2(0, 0);
    for (int b0 = 0; b0 < ntiles; b0 += MESH_TPB * PER) {
        const int t0 = b0 + threadIdx.x * PER;
        int2 v[PER], own = make_int2(0, 0);
#pragma unroll
        for (int q = 0; q < PER; q++) {
            v[q] = t0 + q < ntiles ? tileSums[t0 + q] : make_int2(0, 0);
            own.x += v[q].x;
            own.y += v[q].y;
        }
        int2 tot;
        int2 run = block_scan_int2(own, &tot);
        run.x += carry.x;
        run.y += carry.y;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            if (t0 + q < ntiles) tileSums[t0 + q] = run;
            run.x += v[q].x;
            run.y += v[q].y;
        }
        carry.x += tot.x;
        carry.y += tot.y;
    }
    if (threadIdx.x == 0) {
        totals[0] = carry.x;
        totals[1] = carry.y;
    }
}

// Polygonizer3d::_vertexInterp (polygonizer3d.cpp:455-491): the point where
// the field crosses the threshold on the edge from corner 1 to corner 2,
// kept on the liquid side of a solid crossing.
__device__ void vertex_interp(float p1x, float p1y, float p1z, float p2x, float p2y, float p2z, double v1, double v2,
                              double s1, double s2, float *out) {
    double minmu = 0.0, maxmu = 1.0;
    const double eps = 1e-10;
    if ((s1 < 0.0 && s2 >= 0.0) || (s2 < 0.0 && s1 >= 0.0)) {
        const double diff = s2 - s1;
        if (fabs(diff) > eps) {
            const double su = -s1 / diff;
            if (s1 < 0.0) minmu = su;
            else maxmu = su;
        } else {
            maxmu = minmu;
        }
    }
    minmu = fmax(minmu, eps);
    maxmu = fmin(maxmu, 1.0 - eps);
    double mu = (0.0 - v1) / (v2 - v1);
    if (mu < minmu) mu = minmu;
    if (mu > maxmu) mu = maxmu;
    const float fm = (float)mu;
    out[0] = __fadd_rn(p1x, __fmul_rn(fm, __fsub_rn(p2x, p1x)));
    out[1] = __fadd_rn(p1y, __fmul_rn(fm, __fsub_rn(p2y, p1y)));
    out[2] = __fadd_rn(p1z, __fmul_rn(fm, __fsub_rn(p2z, p1z)));
}

// Numbers the vertices and triangles: the first vertex of every cell that the
// surface cuts, and for each vertex and triangle where it comes from (cell *
// 16 + edge, cell * 16 + number in the cell), as the first two words of the
// place its kernel will fill.  Vertices and triangles are thin on the ground
// (one cell in twenty), so a thread each afterwards keeps the warps full,
// where a kernel over the cells had a few lanes at work.
// With one kernel over the cells for all of it, the numbering and the vertices
// took 1240 us and the triangles 283 us at 128^3, subdivision 2 (209k
// vertices); now 45 us for the numbers, 84 for the vertices, 13 for the
// triangles.
__device__ __forceinline__ void put_origin(int *o, long long code) {
    o[0] = (int)(unsigned)code;
    o[1] = (int)(code >> 32);
}
__device__ __forceinline__ long long get_origin(const int *o) {
    return (long long)((unsigned long long)(unsigned)o[0] | (unsigned long long)(unsigned)o[1] << 32);
}
__global__ void __launch_bounds__(MESH_TPB) k_mesh_number(MeshFrame m, long long ncells, const uint8_t *cube,
                                                          const int2 *tileBase, int *vstart, int *verts, int *tris) {
    const long long base = (long long)blockIdx.x * TILE + (long long)threadIdx.x * CELLS_PER_THREAD;
    const int ci = m.ni - 1, cj = m.nj - 1;
    static_assert(CELLS_PER_THREAD == 8, "a thread's cube indices are one 8-byte word");
    unsigned long long cubes = 0;   // of the thread's cells, those past the end outside
    if (base + CELLS_PER_THREAD <= ncells) {
        cubes = *reinterpret_cast<const unsigned long long *>(cube + base);
    } else {
        for (int q = 0; q < CELLS_PER_THREAD; q++)
            if (base + q < ncells) cubes |= (unsigned long long)cube[base + q] << (8 * q);
    }
    const bool plain = cubes == 0ull || cubes == ~0ull;
    int2 own = make_int2(0, 0);
    if (!plain)
        for (int q = 0; q < CELLS_PER_THREAD; q++) {
            const int cq = (int)(cubes >> (8 * q) & 255);
            if (cq == 0 || cq == 255) continue;
            int i, j, k;
            unflatten(base + q, ci, cj, i, j, k);
            own.x += __popc(cut_mask(cq) & created_mask(i, j, k));
            own.y += tri_count(cq);
        }
    int2 tot;
    int2 run = block_scan_int2(own, &tot);
    if (plain) return;
    const int2 tb = tileBase[blockIdx.x];
    run.x += tb.x;
    run.y += tb.y;
    for (int q = 0; q < CELLS_PER_THREAD; q++) {
        const int cq = (int)(cubes >> (8 * q) & 255);
        if (cq == 0 || cq == 255) continue;
        const long long c = base + q;
        int i, j, k;
        unflatten(c, ci, cj, i, j, k);
        vstart[c] = run.x;
        for (unsigned mk = cut_mask(cq) & created_mask(i, j, k); mk; mk &= mk - 1)
            put_origin(verts + 3LL * run.x++, c * 16 + (__ffs(mk) - 1));
        const int nt = tri_count(cq);
        for (int t = 0; t < nt; t++) put_origin(tris + 3LL * run.y++, c * 16 + t);
    }
}

// The ends of the vertices' edges: their nodes.
__device__ __forceinline__ void edge_end(const MeshFrame &m, long long code, int side, int &a, int &b, int &c) {
    int i, j, k;
    unflatten(code >> 4, m.ni - 1, m.nj - 1, i, j, k);
    const int e = (int)(code & 15), q = side ? kEb[e] : kEa[e];
    a = i + kCx[q];
    b = j + kCy[q];
    c = k + kCz[q];
}
// The ends' field values, a group of lanes each.
template <int GROUP>
__global__ void __launch_bounds__(SEARCH_TPB, 1024 / SEARCH_TPB) k_mesh_ends(ParticleSoA p, const int *cellStart, MeshFrame m,
                                                                             const uint8_t *active, const unsigned *inside,
                                                                             int nverts, const int *origins, float *values) {
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / GROUP;
    if (t >= 2LL * nverts) return;
    int a, b, c;
    edge_end(m, get_origin(origins + 3 * (t >> 1)), (int)(t & 1), a, b, c);
    const float f = node_value<GROUP>(p, cellStart, m, active, inside, a, b, c);
    if (threadIdx.x % GROUP == 0) values[t] = f;
}
// A vertex, moved to the simulation's frame (translate by the chunk offset,
// scale, unscale: particlemesher.cpp:35-55, 271-280).  Apart from the search,
// so that its FP64 work has full warps.
__global__ void __launch_bounds__(MESH_TPB) k_mesh_vertices(MeshFrame m, const float *S, int nverts, const float *values,
                                                            float *verts) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nverts) return;
    float *o = verts + 3LL * t;
    const long long code = get_origin(reinterpret_cast<const int *>(o));
    float x[2], y[2], z[2];
    double sd[2];
    int sign[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        int a, b, c;
        edge_end(m, code, q, a, b, c);
        // Polygonizer3d::_getVertexPosition (polygonizer3d.cpp:356-359)
        x[q] = __fmul_rn(m.subdxf, (float)a);
        y[q] = __fmul_rn(m.subdxf, (float)b);
        z[q] = __fmul_rn(m.subdxf, (float)c);
        sign[q] = solid_sign(m, S, __fadd_rn(x[q], m.offx), __fadd_rn(y[q], m.offy), __fadd_rn(z[q], m.offz));
        sd[q] = (double)sign[q];
    }
    if (sign[0] * sign[1] <= 0)   // the solid's values matter only where the ends' signs differ
        for (int q = 0; q < 2; q++)
            sd[q] = (double)(float)solid_sample(m, S, __fadd_rn(x[q], m.offx), __fadd_rn(y[q], m.offy), __fadd_rn(z[q], m.offz));
    float v[3];
    vertex_interp(x[0], y[0], z[0], x[1], y[1], z[1], (double)values[2LL * t], (double)values[2LL * t + 1], sd[0], sd[1], v);
    o[0] = __fmul_rn(__fmul_rn(__fadd_rn(v[0], m.offx), m.scalef), m.invscalef);
    o[1] = __fmul_rn(__fmul_rn(__fadd_rn(v[1], m.offy), m.scalef), m.invscalef);
    o[2] = __fmul_rn(__fmul_rn(__fadd_rn(v[2], m.offz), m.scalef), m.invscalef);
}

// The vertex on edge e of cell (i, j, k): the cell that creates it, the
// edge's number there, and its rank among that cell's new vertices.
__device__ int edge_vertex(const MeshFrame &m, const uint8_t *cube, const int *vstart, int i, int j, int k, int e) {
    const int o = kEorg[e], d = kEdir[e];
    const int ni = i + kCx[o], nj = j + kCy[o], nk = k + kCz[o];   // the edge's first node
    const int pi = d == 0 ? ni : max(ni - 1, 0), pj = d == 1 ? nj : max(nj - 1, 0), pk = d == 2 ? nk : max(nk - 1, 0);
    const int ox = ni - pi, oy = nj - pj, oz = nk - pk;   // the node's corner offset in the creating cell
    int e2 = 0;
#pragma unroll
    for (int f = 0; f < 12; f++) {
        const int of = kEorg[f];
        if (kEdir[f] == d && kCx[of] == ox && kCy[of] == oy && kCz[of] == oz) e2 = f;
    }
    const long long c2 = (long long)pi + (long long)(m.ni - 1) * ((long long)pj + (long long)(m.nj - 1) * pk);
    const unsigned mk = cut_mask(cube[c2]) & created_mask(pi, pj, pk);
    return vstart[c2] + __popc(mk & ((1u << e2) - 1u));
}

// A triangle (Polygonizer3d::_polygonizeCell, polygonizer3d.cpp:635-656)
__global__ void k_mesh_triangles(MeshFrame m, int ntris, const uint8_t *cube, const int *vstart, int *tris) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntris) return;
    int *o = tris + 3LL * t;
    const long long code = get_origin(o), c = code >> 4;
    int i, j, k;
    unflatten(c, m.ni - 1, m.nj - 1, i, j, k);
    const unsigned w = (unsigned)(kTri[cube[c]] >> (12 * (int)(code & 15)));
#pragma unroll
    for (int q = 0; q < 3; q++) o[q] = edge_vertex(m, cube, vstart, i, j, k, (int)(w >> (4 * q) & 15));
}

// -------------------------------------------------------------- smoothing
// TriangleMesh::_updateVertexTriangles (trianglemesh.cpp:481-499): each
// vertex's triangles in ascending order.
__global__ void k_mesh_adj_count(const int *tris, int ntris, int2 *count) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * ntris) return;
    atomicAdd(&count[tris[t]].x, 1);
}
__global__ void k_mesh_adj_fill(const int *tris, int ntris, const int2 *start, int *cursor, int *list) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * ntris) return;
    const int v = tris[t];
    list[start[v].x + atomicAdd(&cursor[v], 1)] = t / 3;
}
__global__ void k_mesh_adj_sort(const int2 *start, int nverts, int *list) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nverts) return;
    const int b = start[v].x, e = start[v + 1].x;
    for (int a = b + 1; a < e; a++) {
        const int key = list[a];
        int q = a - 1;
        while (q >= b && list[q] > key) {
            list[q + 1] = list[q];
            q--;
        }
        list[q + 1] = key;
    }
}
// TriangleMesh::_smoothTriangleMesh (trianglemesh.cpp:536-570): the mean of
// the other corners of the vertex's triangles, then v + value (mean - v).
__global__ void k_mesh_smooth(const float *vin, float *vout, const int *tris, const int2 *start, const int *list,
                              int nverts, float value) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nverts) return;
    float ax = 0.0f, ay = 0.0f, az = 0.0f;
    int count = 0;
    for (int q = start[v].x; q < start[v + 1].x; q++) {
        const int *t = tris + 3LL * list[q];
        for (int s = 0; s < 3; s++) {
            const int u = t[s];
            if (u == v) continue;
            ax = __fadd_rn(ax, vin[3LL * u]);
            ay = __fadd_rn(ay, vin[3LL * u + 1]);
            az = __fadd_rn(az, vin[3LL * u + 2]);
            count++;
        }
    }
    const float inv = (float)(1.0 / (double)(float)count);   // vec3 operator/= (vmath.cpp:105-111)
    ax = __fmul_rn(ax, inv);
    ay = __fmul_rn(ay, inv);
    az = __fmul_rn(az, inv);
    const float x = vin[3LL * v], y = vin[3LL * v + 1], z = vin[3LL * v + 2];
    vout[3LL * v] = __fadd_rn(x, __fmul_rn(value, __fsub_rn(ax, x)));
    vout[3LL * v + 1] = __fadd_rn(y, __fmul_rn(value, __fsub_rn(ay, y)));
    vout[3LL * v + 2] = __fadd_rn(z, __fmul_rn(value, __fsub_rn(az, z)));
}

// ------------------------------------------------------------------ scans
// Exclusive scan of n int2 values into out[0..n] (out[n] = the totals), by
// tiles of TILE: tile sums, their scan in one CTA, then each tile again.
__global__ void __launch_bounds__(MESH_TPB) k_scan2_tiles(const int2 *in, long long n, int2 *tileSums) {
    const long long base = (long long)blockIdx.x * TILE + (long long)threadIdx.x * CELLS_PER_THREAD;
    int2 own = make_int2(0, 0);
    for (int q = 0; q < CELLS_PER_THREAD; q++)
        if (base + q < n) {
            own.x += in[base + q].x;
            own.y += in[base + q].y;
        }
    int2 tot;
    block_scan_int2(own, &tot);
    if (threadIdx.x == 0) tileSums[blockIdx.x] = tot;
}
__global__ void __launch_bounds__(MESH_TPB) k_scan2_apply(const int2 *in, long long n, const int2 *tileBase,
                                                          const int *totals, int2 *out) {
    const long long base = (long long)blockIdx.x * TILE + (long long)threadIdx.x * CELLS_PER_THREAD;
    int2 own = make_int2(0, 0);
    for (int q = 0; q < CELLS_PER_THREAD; q++)
        if (base + q < n) {
            own.x += in[base + q].x;
            own.y += in[base + q].y;
        }
    int2 tot;
    int2 run = block_scan_int2(own, &tot);
    run.x += tileBase[blockIdx.x].x;
    run.y += tileBase[blockIdx.x].y;
    for (int q = 0; q < CELLS_PER_THREAD; q++) {
        const long long t = base + q;
        if (t >= n) break;
        const int2 v = in[t];
        out[t] = run;
        run.x += v.x;
        run.y += v.y;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = make_int2(totals[0], totals[1]);
}

template <class T>
int grow(MeshBuffers &mb, T **p, long long *cap, long long need) {
    if (need <= *cap && *p) return FLIP_OK;
    if (*p) {
        cudaFree(*p);
        mb.bytes -= (long long)sizeof(T) * *cap;
        *p = nullptr;
        *cap = 0;
    }
    const long long want = std::max<long long>(need + need / 4, 1);
    cudaError_t e = cudaMalloc((void **)p, (size_t)want * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return record_error(FLIP_E_NOMEM, std::string("surface mesh buffers: ") + cudaGetErrorString(e));
    }
    *cap = want;
    mb.bytes += (long long)sizeof(T) * want;
    return FLIP_OK;
}

#define MCK(call)                                                                                         \
    do {                                                                                                  \
        cudaError_t e_ = (call);                                                                          \
        if (e_ != cudaSuccess) return record_error(FLIP_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)
#define MRC(call)                  \
    do {                           \
        int rc_ = (call);          \
        if (rc_) return rc_;       \
    } while (0)

}  // namespace

void mesh_release(MeshBuffers &mb) {
    void *ptrs[] = {mb.occ, mb.active, mb.inside, mb.occupied, mb.cube, mb.vstart, mb.tiles, mb.totals,
                    mb.verts[0], mb.verts[1], mb.tris, mb.adj, mb.adjStart, mb.adjCursor, mb.adjList};
    for (void *q : ptrs)
        if (q) cudaFree(q);
    mb = MeshBuffers{};
}

int mesh_surface(const MeshJob &job, MeshBuffers &mb, cudaStream_t s) {
    const StepConsts &c = job.c;
    mb.nverts = mb.ntris = 0;
    mb.cur = 0;
    if (job.n <= 0) return FLIP_OK;   // no particles: an empty mesh (fluidsimulation.cpp:5047-5051)
    const int sd = job.subdivisions;
    MeshFrame m{};
    m.I = c.I;
    m.J = c.J;
    m.K = c.K;
    m.dx = c.dx;
    m.invdx = 1.0 / c.dx;
    m.subdx = c.dx / (double)sd;
    m.invsub = 1.0 / m.subdx;
    m.invsubf = (float)m.invsub;
    m.dxf = (float)m.dx;
    m.invdxf = (float)m.invdx;
    m.subdxf = (float)m.subdx;
    for (int a = 0; a < MB; a++) m.nodePos[a] = (float)((double)(float)a * m.subdx);
    m.blockdx = MB * m.subdx;
    m.invBlock = 1.0 / m.blockdx;
    m.invBlockf = (float)m.invBlock;
    m.blockdxF = (float)(MB * m.subdx);
    m.invBlockF = 1.0 / (double)m.blockdxF;
    m.invBlockFf = (float)m.invBlockF;
    m.r = (float)job.radius;
    m.sr = 1.5f * m.r;   // _searchRadiusFactor * r (particlemesher.h:193)
    m.maxd = (float)(3.0 * job.radius);
    const int sI = c.I * sd + 1, sJ = c.J * sd + 1, sK = c.K * sd + 1;
    m.nbI = (sI + MB - 1) / MB;
    m.nbJ = (sJ + MB - 1) / MB;
    m.nbK = (sK + MB - 1) / MB;
    const long long nb = (long long)m.nbI * m.nbJ * m.nbK;

    // blocks that hold particles, feathered by one block
    MRC(grow(mb, &mb.occ, &mb.occCap, nb));
    MCK(cudaMemsetAsync(mb.occ, 0, nb, s));
    { FLIP_COUNT(1); k_mesh_occupancy<<<div_up(job.n, MESH_TPB), MESH_TPB, 0, s>>>(job.p, job.n, m, mb.occ); }
    std::vector<uint8_t> occ(nb), act(nb, 0);
    MCK(cudaMemcpyAsync(occ.data(), mb.occ, nb, cudaMemcpyDeviceToHost, s));
    FLIP_SYNC_COUNT();
    MCK(cudaStreamSynchronize(s));
    auto bidx = [&](int a, int b, int e) { return a + (long long)m.nbI * (b + (long long)m.nbJ * e); };
    for (int e = 0; e < m.nbK; e++)
        for (int b = 0; b < m.nbJ; b++)
            for (int a = 0; a < m.nbI; a++) {
                if (!occ[bidx(a, b, e)]) continue;
                for (int z = std::max(e - 1, 0); z <= std::min(e + 1, m.nbK - 1); z++)
                    for (int y = std::max(b - 1, 0); y <= std::min(b + 1, m.nbJ - 1); y++)
                        for (int x = std::max(a - 1, 0); x <= std::min(a + 1, m.nbI - 1); x++) act[bidx(x, y, z)] = 1;
            }
    // the one compute chunk (particlemesher.cpp:139-282)
    int lo[3] = {m.nbI, m.nbJ, m.nbK}, hi[3] = {0, 0, 0};
    const int nbd[3] = {m.nbI, m.nbJ, m.nbK};
    bool any = false;
    for (int e = 0; e < m.nbK; e++)
        for (int b = 0; b < m.nbJ; b++)
            for (int a = 0; a < m.nbI; a++)
                if (act[bidx(a, b, e)]) {
                    any = true;
                    const int g[3] = {a, b, e};
                    for (int d = 0; d < 3; d++) {
                        lo[d] = std::min(lo[d], g[d]);
                        hi[d] = std::max(hi[d], g[d] + 1);
                    }
                }
    if (!any) return FLIP_OK;
    int split = 0;
    if (m.nbJ > m.nbI) split = 1;
    if (m.nbK > nbd[split]) split = 2;
    for (int d = 0; d < 3; d++)
        if (d != split) {
            lo[d] = std::max(lo[d] - 1, 0);
            hi[d] = std::min(hi[d] + 1, nbd[d]);
        }
    const int sub[3] = {sI, sJ, sK};
    int gmin[3], gmax[3];
    for (int d = 0; d < 3; d++) {
        gmin[d] = MB * lo[d];
        gmax[d] = std::min(MB * hi[d], sub[d]);
    }
    m.ni = gmax[0] - gmin[0];
    m.nj = gmax[1] - gmin[1];
    m.nk = gmax[2] - gmin[2];
    m.cbI = hi[0] - lo[0];
    m.cbJ = hi[1] - lo[1];
    m.cbK = hi[2] - lo[2];
    m.offx = (float)((double)(float)gmin[0] * m.subdx);   // Grid3d::GridIndexToPosition
    m.offy = (float)((double)(float)gmin[1] * m.subdx);
    m.offz = (float)((double)(float)gmin[2] * m.subdx);
    // AABB(pmin, pmax).expand(2 (r + 1e-6)) (particlemesher.cpp:287-292, aabb.cpp:40-52, 122-128)
    {
        const float pmx = (float)((double)(float)gmax[0] * m.subdx), pmy = (float)((double)(float)gmax[1] * m.subdx),
                    pmz = (float)((double)(float)gmax[2] * m.subdx);
        const double v = 2.0f * (job.radius + (double)1e-6f), h = 0.5 * v;
        m.bbx = m.offx - (float)h;
        m.bby = m.offy - (float)h;
        m.bbz = m.offz - (float)h;
        // a coordinate p is inside where (double)p < bb + extent: where p is
        // below the smallest float that is no less
        auto upper = [](double x) {
            const float f = (float)x;
            return (double)f < x ? std::nextafter(f, INFINITY) : f;
        };
        m.bhx = upper((double)m.bbx + (((double)pmx - (double)m.offx) + v));
        m.bhy = upper((double)m.bby + (((double)pmy - (double)m.offy) + v));
        m.bhz = upper((double)m.bbz + (((double)pmz - (double)m.offz) + v));
    }
    // how ScalarField::setSolidSDF finds solid nodes (scalarfield.cpp:372-395)
    const float offLen = std::sqrt(m.offx * m.offx + m.offy * m.offy + m.offz * m.offz);
    if (m.ni == c.I + 1 && m.nj == c.J + 1 && m.nk == c.K + 1 && std::fabs(m.subdx - c.dx) < 1e-12)
        m.solidMode = 2;
    else if (std::fabs(2 * m.subdx - c.dx) < 1e-6 && offLen < 1e-6)
        m.solidMode = 1;
    else
        m.solidMode = 0;
    const double scale = 0.1 / m.subdx;   // _localdx / _subdx (particlemesher.cpp:40-52)
    m.scalef = (float)scale;
    m.invscalef = (float)(1.0 / scale);

    const long long ncb = (long long)m.cbI * m.cbJ * m.cbK;
    // the chunk's blocks: their frames' origins along each axis, then which are active
    const int nb1[3] = {m.cbI, m.cbJ, m.cbK};
    // the rows of cells that a search visits, nearest first, for a node nearer
    // to the lower side of its cell in y and z
    m.reach = m.sr + 1.02f * m.subdxf;
    m.signReach = std::min(m.r * 1.001f, m.reach);
    m.slack = 0.01f * m.dxf * (m.dxf + m.reach);
    m.near2 = std::max(m.sr - 0.02f * m.subdxf, 0.0f) * std::max(m.sr - 0.02f * m.subdxf, 0.0f);
    std::vector<MeshRow> rows;
    const int R2 = (int)std::ceil(m.reach * m.invdxf + 0.02f);
    auto side = [](int o) { return o == 0 ? 0.0f : (o > 0 ? o - 1.0f : -o - 0.5f); };   // at least so far, in cells
    for (int z = -std::min(R2, c.K); z <= std::min(R2, c.K); z++)
        for (int y = -std::min(R2, c.J); y <= std::min(R2, c.J); y++) {
            const float dy = std::max(side(y) - 0.01f, 0.0f) * m.dxf, dz = std::max(side(z) - 0.01f, 0.0f) * m.dxf;
            rows.push_back({dy * dy + dz * dz, (short)y, (short)z});
        }
    std::stable_sort(rows.begin(), rows.end(), [&](const MeshRow &a, const MeshRow &b) {
        return a.least != b.least ? a.least < b.least
                                  : std::abs(a.y) + std::abs(a.z) < std::abs(b.y) + std::abs(b.z);
    });
    m.nrows = (int)rows.size();
    const size_t rowBytes = rows.size() * sizeof(MeshRow);
    const size_t tables = rowBytes + sizeof(float) * ((size_t)m.cbI + m.cbJ + m.cbK);
    std::vector<uint8_t> blocks(tables + ncb);
    uint8_t *cact = blocks.data() + tables;
    for (int d = 0, at = 0; d < 3; at += nb1[d++])
        for (int b = 0; b < nb1[d]; b++) {
            const float o = (float)((double)(float)b * m.blockdx);
            std::memcpy(blocks.data() + rowBytes + sizeof(float) * (at + b), &o, sizeof(o));
        }
    std::memcpy(blocks.data(), rows.data(), rowBytes);
    for (int e = 0; e < m.cbK; e++)
        for (int b = 0; b < m.cbJ; b++)
            for (int a = 0; a < m.cbI; a++)
                cact[a + (long long)m.cbI * (b + (long long)m.cbJ * e)] = act[bidx(a + lo[0], b + lo[1], e + lo[2])];
    m.wpr = (m.ni + 31) / 32;
    const long long nwords = (long long)m.wpr * m.nj * m.nk;
    const long long ncells = (long long)(m.ni - 1) * (m.nj - 1) * (m.nk - 1);
    const long long ntiles = std::max<long long>((ncells + TILE - 1) / TILE, 1);
    MRC(grow(mb, &mb.active, &mb.activeCap, (long long)blocks.size()));
    MRC(grow(mb, &mb.inside, &mb.insideCap, nwords));
    MRC(grow(mb, &mb.cube, &mb.cubeCap, std::max<long long>(ncells, 1)));
    MRC(grow(mb, &mb.vstart, &mb.vstartCap, std::max<long long>(ncells, 1)));
    MRC(grow(mb, &mb.tiles, &mb.tilesCap, ntiles));
    MRC(grow(mb, &mb.totals, &mb.totalsCap, 2));
    MCK(cudaMemcpyAsync(mb.active, blocks.data(), blocks.size(), cudaMemcpyHostToDevice, s));
    m.rows = reinterpret_cast<const MeshRow *>(mb.active);
    m.blockPos[0] = reinterpret_cast<const float *>(mb.active + rowBytes);
    m.blockPos[1] = m.blockPos[0] + m.cbI;
    m.blockPos[2] = m.blockPos[1] + m.cbJ;
    const uint8_t *active = mb.active + tables;
    // no farther than the word of cells beside a cell's own
    const int R = (int)std::ceil(m.signReach * m.invdxf + 0.02f);
    unsigned *around = nullptr;
    if (R < 32) {
        m.wpc = (c.I + 31) / 32;
        const long long cw = (long long)m.wpc * c.J * c.K;
        MRC(grow(mb, &mb.occupied, &mb.occupiedCap, 2 * cw));
        around = mb.occupied + cw;
        { FLIP_COUNT(1); k_mesh_occupied<<<div_up(cw, MESH_TPB / 32), MESH_TPB, 0, s>>>(job.cellStart, m, mb.occupied); }
        { FLIP_COUNT(1); k_mesh_around<<<div_up(cw, MESH_TPB), MESH_TPB, 0, s>>>(m, mb.occupied, R, around); }
    }
    // the list of wall nodes lies where vstart will
    const int room = (int)std::min<long long>(mb.vstartCap, 0x7fffffff);
    MCK(cudaMemsetAsync(mb.totals, 0, sizeof(int), s));
    {
        FLIP_COUNT(1);
        k_mesh_inside<<<div_up(nwords, SEARCH_TPB / 32), SEARCH_TPB, 0, s>>>(job.p, job.cellStart, m, active, around, job.solidPhi,
                                                                              mb.inside, mb.vstart, room, mb.totals);
    }
    { FLIP_COUNT(1); k_mesh_walls<<<152, MESH_TPB, 0, s>>>(m, job.solidPhi, mb.vstart, room, mb.totals, mb.inside); }
    if (ncells <= 0) return FLIP_OK;
    { FLIP_COUNT(1); k_mesh_count<<<(unsigned)ntiles, MESH_TPB, 0, s>>>(m, mb.inside, ncells, mb.cube, mb.tiles); }
    { FLIP_COUNT(1); k_mesh_scan_tiles<<<1, MESH_TPB, 0, s>>>(mb.tiles, (int)ntiles, mb.totals); }
    int totals[2];
    MCK(cudaMemcpyAsync(totals, mb.totals, sizeof(totals), cudaMemcpyDeviceToHost, s));
    FLIP_SYNC_COUNT();
    MCK(cudaStreamSynchronize(s));
    const int nverts = totals[0], ntris = totals[1];
    if (nverts <= 0 || ntris <= 0) return FLIP_OK;
    MRC(grow(mb, &mb.verts[0], &mb.vertsCap[0], 3LL * nverts));
    MRC(grow(mb, &mb.verts[1], &mb.vertsCap[1], 3LL * nverts));
    MRC(grow(mb, &mb.tris, &mb.trisCap, 3LL * ntris));
    {
        FLIP_COUNT(1);
        k_mesh_number<<<(unsigned)ntiles, MESH_TPB, 0, s>>>(m, ncells, mb.cube, mb.tiles, mb.vstart,
                                                             reinterpret_cast<int *>(mb.verts[0]), mb.tris);
    }
    {
        // few vertices: more lanes to a search, which then ends sooner (12650
        // vertices: 112 us with eight, 163 with four); many: fewer, which look
        // at less (208844: 245 us with eight, 174 with four)
        auto ends = [&](auto kernel, int group) {
            FLIP_COUNT(1);
            kernel<<<div_up(2LL * group * nverts, SEARCH_TPB), SEARCH_TPB, 0, s>>>(
                job.p, job.cellStart, m, active, mb.inside, nverts, reinterpret_cast<const int *>(mb.verts[0]), mb.verts[1]);
        };
        if (nverts < 65536) ends(k_mesh_ends<8>, 8);
        else ends(k_mesh_ends<4>, 4);
    }
    { FLIP_COUNT(1); k_mesh_vertices<<<div_up(nverts, MESH_TPB), MESH_TPB, 0, s>>>(m, job.solidPhi, nverts, mb.verts[1], mb.verts[0]); }
    { FLIP_COUNT(1); k_mesh_triangles<<<div_up(ntris, MESH_TPB), MESH_TPB, 0, s>>>(m, ntris, mb.cube, mb.vstart, mb.tris); }
    mb.nverts = nverts;
    mb.ntris = ntris;
    if (job.smoothIterations > 0) {
        // TriangleMesh::smooth (trianglemesh.cpp:572-583)
        const long long vt = (nverts + TILE - 1) / TILE;
        MRC(grow(mb, &mb.adj, &mb.adjCap, (long long)nverts));
        MRC(grow(mb, &mb.adjStart, &mb.adjStartCap, (long long)nverts + 1));
        MRC(grow(mb, &mb.adjCursor, &mb.adjCursorCap, (long long)nverts));
        MRC(grow(mb, &mb.adjList, &mb.adjListCap, 3LL * ntris));
        MRC(grow(mb, &mb.tiles, &mb.tilesCap, std::max(ntiles, vt)));
        MCK(cudaMemsetAsync(mb.adj, 0, (size_t)nverts * sizeof(int2), s));
        MCK(cudaMemsetAsync(mb.adjCursor, 0, (size_t)nverts * sizeof(int), s));
        { FLIP_COUNT(1); k_mesh_adj_count<<<div_up(3LL * ntris, MESH_TPB), MESH_TPB, 0, s>>>(mb.tris, ntris, mb.adj); }
        { FLIP_COUNT(1); k_scan2_tiles<<<(unsigned)vt, MESH_TPB, 0, s>>>(mb.adj, nverts, mb.tiles); }
        { FLIP_COUNT(1); k_mesh_scan_tiles<<<1, MESH_TPB, 0, s>>>(mb.tiles, (int)vt, mb.totals); }
        { FLIP_COUNT(1); k_scan2_apply<<<(unsigned)vt, MESH_TPB, 0, s>>>(mb.adj, nverts, mb.tiles, mb.totals, mb.adjStart); }
        { FLIP_COUNT(1); k_mesh_adj_fill<<<div_up(3LL * ntris, MESH_TPB), MESH_TPB, 0, s>>>(mb.tris, ntris, mb.adjStart, mb.adjCursor, mb.adjList); }
        { FLIP_COUNT(1); k_mesh_adj_sort<<<div_up(nverts, MESH_TPB), MESH_TPB, 0, s>>>(mb.adjStart, nverts, mb.adjList); }
        const float value = (float)job.smoothValue;
        for (int it = 0; it < job.smoothIterations; it++) {
            FLIP_COUNT(1);
            k_mesh_smooth<<<div_up(nverts, MESH_TPB), MESH_TPB, 0, s>>>(mb.verts[mb.cur], mb.verts[mb.cur ^ 1], mb.tris,
                                                                       mb.adjStart, mb.adjList, nverts, value);
            mb.cur ^= 1;
        }
    }
    MCK(cudaGetLastError());
    return FLIP_OK;
}

}  // namespace flip
