// Uniform 2-D AST smoke solver on the GPU: the reference's ASTSolver<2> (include/ast_solver.h), the
// solver behind its Python module's ASTSolver2.  Storage follows the reference's grids (x fastest):
// cells x + y*nx, vertices (tilted cells) x + y*(nx+1), x faces x + y*(nx+1), y faces x + y*nx, four
// tilted-face velocities per vertex.  The reference is configured with CORRECTION_MAC and
// LAYOUT_ADJUST_DENSITY on and EDGE_NODE_ADAPTIVITY off (include/ast_general.h:9-13), so edge nodes
// never open and the degrees of freedom are the cells and the open tilts.
//
// Every floating-point expression keeps the reference's operand order and the library is built
// with FMA contraction off, so each stage reproduces the CPU restatement bit for bit.  One change
// of evaluation, not of arithmetic: ASTFaceGrid<double, 2>::sample's correction term
// (include/ast_face_grid.h:59-63) is an `auto` Eigen expression that refers to a temporary destroyed
// before it is read, so the reference's own build reads a dead stack slot there; this code
// evaluates the difference the expression spells out.
//
// Kernels per sub-step: source, force (+ x walls), numbering (scan of the open tilts), assembly of
// padded rows -> CSR (shared with the octree path), MIC(0) factorisation and PCG (shared; the
// preconditioner is the wavefront kernel below), pressure correction (+ x walls), dual velocities,
// and one fused advection kernel (layout adjustment, density, heat, tilted faces and MAC faces;
// density and heat share each back-trace).
#include <cstdint>
#include <type_traits>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "astg_launch.h"
#include "astg2d_launch.h"

namespace cg = cooperative_groups;

namespace astg {
namespace g2 {

constexpr double SQRT2 = 1.4142135623730951;   // include/macro.h:16
constexpr double INV_SQRT2 = 1.0 / SQRT2;       // include/macro.h:19 (value of the macro)
constexpr double EPS2 = 2.220446049250313e-16;  // include/general.h:48
constexpr int TB2 = 256;

// include/ast_constant.h:24-26 and include/constants.h:36-39 (the same values)
__constant__ double TILT_OFF[4][2] = {{INV_SQRT2, INV_SQRT2}, {INV_SQRT2, -INV_SQRT2},
                                      {-INV_SQRT2, -INV_SQRT2}, {-INV_SQRT2, INV_SQRT2}};
// include/ast_constant.h:39-44 (mac_direction: 0 x+, 1 x-, 2 y+, 3 y-)
__constant__ int TILT_MAC[4][2] = {{0, 2}, {0, 3}, {1, 3}, {1, 2}};
// include/constants.h:71-77
__constant__ int OCT_NB_TILT[4][2] = {{1, 1}, {1, 0}, {0, 0}, {0, 1}};
__constant__ int TILT_NB_OCT[4][2] = {{0, 0}, {0, -1}, {-1, -1}, {-1, 0}};

struct P2 {
    double x, y;
};

static inline int nblk2(long long n) { return (int)((n + TB2 - 1) / TB2); }
__device__ inline double dmin2(double a, double b) { return (b < a) ? b : a; }  // std::min
__device__ inline double lerp2(double a, double b, double f) { return a * (1 - f) + b * f; }
// include/util.h:172-176
__device__ inline double bilerp2(double v00, double v01, double v11, double v10, double fx, double fy) {
    return lerp2(lerp2(v00, v10, fx), lerp2(v01, v11, fx), fy);
}
// include/util.h:243-256, one component: truncating cast, index clamped to [0, high - 1], fraction
// clamped to [0, 1]
__device__ inline void bary2(double x, int high, int* i, double* f) {
    int c = (int)x;
    c = c < 0 ? 0 : c;
    c = c > high - 1 ? high - 1 : c;
    *i = c;
    double t = x - c;
    t = t < 0.0 ? 0.0 : t;
    *f = t > 1.0 ? 1.0 : t;
}

__device__ inline int ci(const Grid2& g, int x, int y) { return x + y * g.nx; }
__device__ inline int vi(const Grid2& g, int x, int y) { return x + y * (g.nx + 1); }
__device__ inline int mxi(const Grid2& g, int x, int y) { return x + y * (g.nx + 1); }
__device__ inline int myi(const Grid2& g, int x, int y) { return x + y * g.nx; }
// CellCenteredGrid::position, VertexCenteredGrid::position, FaceCenteredGrid::position
__device__ inline P2 cellPos(const Grid2& g, int x, int y) { return P2{(x + 0.5) * g.dx, (y + 0.5) * g.dx}; }
__device__ inline P2 vertPos(const Grid2& g, int x, int y) { return P2{x * g.dx, y * g.dx}; }
__device__ inline P2 macPos(const Grid2& g, int a, int x, int y) {
    return a == 0 ? P2{(x + 0.0) * g.dx, (y + 0.5) * g.dx} : P2{(x + 0.5) * g.dx, (y + 0.0) * g.dx};
}
__device__ inline bool inSphere(P2 p) {
    double ax = p.x - 0.5, ay = p.y - 0.04;  // sphereSource2DSetup: centre (0.5, 0.04), radius 0.03
    return sqrt(ax * ax + ay * ay) < 0.03;
}

// CellCenteredGrid<T, 2>::sample (include/cell_centered_grid.h:40-55)
__device__ inline double cellSample(const Grid2& g, const double* c, P2 pos) {
    int ix, iy;
    double fx, fy;
    bary2(pos.x / g.dx - 0.5, g.nx - 1, &ix, &fx);
    bary2(pos.y / g.dx - 0.5, g.ny - 1, &iy, &fy);
    int x1 = min(ix + 1, g.nx - 1), y1 = min(iy + 1, g.ny - 1);
    return bilerp2(c[ci(g, ix, iy)], c[ci(g, ix, y1)], c[ci(g, x1, y1)], c[ci(g, x1, iy)], fx, fy);
}
// ASTGrid<T, 2>::sample2D (include/ast_grid.h:62-96) with the edge nodes closed
__device__ inline double scalarSample(const Grid2& g, const double* c, const double* v, const uint8_t* open, P2 pos) {
    int cx, cy;
    double fx, fy;
    bary2(pos.x / g.hdx, g.nx * 2, &cx, &fx);
    bary2(pos.y / g.hdx, g.ny * 2, &cy, &fy);
    cx = cx < 1 ? 1 : cx;
    cy = cy < 1 ? 1 : cy;
    int bx = (cx - 1) / 2, by = (cy - 1) / 2;
    int tx = bx + 1, ty = by + 1;
    if (!open[vi(g, tx, ty)]) return cellSample(g, c, pos);
    int ox = min(bx * 2 + 1 - cx, 0), oy = min(by * 2 + 1 - cy, 0);
    fx = fx / 2.0 - 0.5 * (double)ox;
    fy = fy / 2.0 - 0.5 * (double)oy;
    int b1x = min(tx, g.nx - 1), b1y = min(ty, g.ny - 1);
    double v0 = c[ci(g, bx, by)], v1 = c[ci(g, bx, b1y)], v2 = c[ci(g, b1x, b1y)], v3 = c[ci(g, b1x, by)];
    double val = bilerp2(v0, v1, v2, v3, fx, fy);
    double delta = v[vi(g, tx, ty)] - 0.25 * (v0 + v1 + v2 + v3);
    return val + 2 * delta * dmin2(dmin2(fx, fy), dmin2(1 - fx, 1 - fy));
}
// FaceCenteredGrid<Real, 2>::sampleComponent (include/face_centered_grid.h:43-60)
__device__ inline double macAxis(const Grid2& g, const double* mx, const double* my, int a, P2 pos) {
    double rx = pos.x / g.dx, ry = pos.y / g.dx;
    if (a == 0) ry = ry - 0.5;
    else rx = rx - 0.5;
    int lx = g.nx - 1 + (a == 0), ly = g.ny - 1 + (a == 1);
    int ix, iy;
    double fx, fy;
    bary2(rx, lx, &ix, &fx);
    bary2(ry, ly, &iy, &fy);
    int x1 = min(ix + 1, lx), y1 = min(iy + 1, ly);
    if (a == 0)
        return bilerp2(mx[mxi(g, ix, iy)], mx[mxi(g, ix, y1)], mx[mxi(g, x1, y1)], mx[mxi(g, x1, iy)], fx, fy);
    return bilerp2(my[myi(g, ix, iy)], my[myi(g, ix, y1)], my[myi(g, x1, y1)], my[myi(g, x1, iy)], fx, fy);
}
// ASTFaceGrid<Real, 2>::sample with CORRECTION_MAC (include/ast_face_grid.h:52-66), the correction
// term evaluated
__device__ inline P2 velSample(const Grid2& g, const Fields2& F, const double* dual, P2 pos) {
    int ix, iy;
    double fx, fy;
    bary2(pos.x / g.dx - 0.5, g.nx - 1, &ix, &fx);
    bary2(pos.y / g.dx - 0.5, g.ny - 1, &iy, &fy);
    P2 ret{macAxis(g, F.mx, F.my, 0, pos), macAxis(g, F.mx, F.my, 1, pos)};
    int v = vi(g, ix + 1, iy + 1);
    if (!F.open[v]) return ret;
    P2 vp{(ix + 1) * g.dx, (iy + 1) * g.dx};
    double ddx = dual[2 * v] - macAxis(g, F.mx, F.my, 0, vp);
    double ddy = dual[2 * v + 1] - macAxis(g, F.mx, F.my, 1, vp);
    double m = dmin2(dmin2(fx, fy), dmin2(1 - fx, 1 - fy));
    return P2{ret.x + 2 * ddx * m, ret.y + 2 * ddy * m};
}
// backTrace (include/ast_advection.h:11-16)
__device__ inline P2 backTrace(const Grid2& g, const Fields2& F, const double* dual, P2 p, double dt) {
    P2 v = velSample(g, F, dual, p);
    P2 mid{p.x - v.x * dt * 0.5, p.y - v.y * dt * 0.5};
    P2 w = velSample(g, F, dual, mid);
    return P2{p.x - w.x * dt, p.y - w.y * dt};
}

// ------------------------------------------------------------------ source, force
// sphereSource2DSetup (include/ast_solver.h:148-205): density and heat 1 on every cell and vertex
// inside the sphere, the open tilts inside it take (1, -1, 1, -1) / sqrt(2), the y faces 1
__global__ void k2_source(Grid2 g, Fields2 F) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nc = g.nx * g.ny, nv = (g.nx + 1) * (g.ny + 1), nmy = g.nx * (g.ny + 1);
    if (i < nc && inSphere(cellPos(g, i % g.nx, i / g.nx))) {
        F.dC[i] = 1;
        F.hC[i] = 1;
    }
    if (i < nv && inSphere(vertPos(g, i % (g.nx + 1), i / (g.nx + 1)))) {
        F.dV[i] = 1;
        F.hV[i] = 1;
        if (F.open[i]) {
            F.tv[4 * i + 0] = INV_SQRT2 * 1.0;
            F.tv[4 * i + 1] = -INV_SQRT2 * 1.0;
            F.tv[4 * i + 2] = INV_SQRT2 * 1.0;
            F.tv[4 * i + 3] = -INV_SQRT2 * 1.0;
        }
    }
    if (i < nmy && inSphere(macPos(g, 1, i % g.nx, i / g.nx))) F.my[i] = 1.0;
}
// addForce (include/ast_solver.h:246-281) with constrainVelocity (:609-616): the open tilts take
// beta dt times the heat sampled half a cell out along each tilted normal, projected on the
// upward axis; the y faces take beta dt times the heat at the face; the x walls are closed
__global__ void k2_force(Grid2 g, Fields2 F, double dt) {
    const double beta = 0.5;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nv = (g.nx + 1) * (g.ny + 1), nmy = g.nx * (g.ny + 1);
    if (i < nv && F.open[i]) {
        P2 pc = vertPos(g, i % (g.nx + 1), i / (g.nx + 1));
        double f[4];
        for (int k = 0; k < 4; ++k) {
            P2 p{pc.x + TILT_OFF[k][0] * g.hdx, pc.y + TILT_OFF[k][1] * g.hdx};
            f[k] = scalarSample(g, F.hC, F.hV, F.open, p) * ((k & 1) ? -INV_SQRT2 : INV_SQRT2);
        }
        for (int k = 0; k < 4; ++k) F.tv[4 * i + k] += f[k] * beta * dt;
    }
    if (i < nmy) F.my[i] += scalarSample(g, F.hC, F.hV, F.open, macPos(g, 1, i % g.nx, i / g.nx)) * beta * dt;
    if (i < g.ny) {
        F.mx[mxi(g, 0, i)] = 0;
        F.mx[mxi(g, g.nx, i)] = 0;
    }
}

// ------------------------------------------------------------------ numbering
// updateIndex (include/ast_solver.h:585-607): cells keep 0 .. nc-1, the open tilts follow in
// vertex order
__global__ void k2_count(Grid2 g, const uint8_t* open, int* cnt) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (g.nx + 1) * (g.ny + 1)) cnt[i] = open[i] ? 1 : 0;
}
__global__ void k2_assign(Grid2 g, const uint8_t* open, const int* base, const int* total, int* vIdx, int* nDof) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nc = g.nx * g.ny;
    if (i < (g.nx + 1) * (g.ny + 1)) vIdx[i] = open[i] ? nc + base[i] : -1;
    if (i == 0) *nDof = nc + *total;
}

// ------------------------------------------------------------------ assembly
// project's system (include/ast_solver.h:326-469).  Cell rows: the open tilts at the cell's corners
// (coefficient 1, the tilt's face takes half of each of the two MAC faces it cuts), then the MAC
// faces with what is left of their area (Neumann x walls, Dirichlet top and bottom); the centre and
// the right-hand side accumulate in the reference's order, the entries are written sorted by
// column (cells below, the diagonal, cells above, then the tilts, whose indices follow the cells').
__global__ void k2_asm_cell(Grid2 g, Dev d, Fields2 F, const int* vIdx, Proj P) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = g.nx, ny = g.ny;
    if (c >= nx * ny) return;
    const int x = c % nx, y = c / nx;
    bool ok[4], fent[4] = {false, false, false, false};
    int tIdx[4] = {0, 0, 0, 0};
    double tcoef[4] = {0, 0, 0, 0}, fcoef[4] = {0, 0, 0, 0};
    double fa[4] = {0, 0, 0, 0}, center = 0, tb = 0;
    for (int k = 0; k < 4; ++k) {
        const int v = vi(g, x + OCT_NB_TILT[k][0], y + OCT_NB_TILT[k][1]);
        ok[k] = F.open[v] != 0;
        if (!ok[k]) continue;
        for (int i = 0; i < 2; ++i) fa[TILT_MAC[k][i]] -= g.hdx;
        tIdx[k] = vIdx[v];
        if (tIdx[k] < 0) report(d, DS_MISSING_NODE);
        double area = g.hdx * SQRT2 * (1.0 - 0.5 * 0.0);
        double coeff = area / g.tiltOctDx;
        tcoef[k] = -coeff;
        center += coeff;
        int sign = k <= 1 ? -1 : 1;
        tb += sign * area * F.tv[4 * v + (k + 2) % 4];
    }
    for (int k = 0; k < 4; ++k) {
        fa[k] += g.dx;
        if (!(fa[k] > EPS2)) continue;
        const int axis = k / 2;
        int nbx = x, nby = y;
        if (axis == 0) nbx += (k & 1) ? -1 : 1;
        else nby += (k & 1) ? -1 : 1;
        const int fx = x + (axis == 0 && !(k & 1)), fy = y + (axis == 1 && !(k & 1));
        const double u = axis == 0 ? F.mx[mxi(g, fx, fy)] : F.my[myi(g, fx, fy)];
        const bool valid = nbx >= 0 && nby >= 0 && nbx < nx && nby < ny;
        if (valid || axis == 1) {
            double coeff = fa[k] / g.dx;
            if (valid) {
                fent[k] = true;
                fcoef[k] = -coeff;
            }
            center += coeff;
            tb += ((k & 1) ? 1 : -1) * fa[k] * u;
        }
    }
    if (center < EPS2) center = 1;
    const size_t o = (size_t)c * ROW_W;
    int n = 0;
    auto put = [&](int col, double v) {
        P.padCol[o + n] = col;
        P.padVal[o + n] = v;
        ++n;
    };
    if (fent[3]) put(c - nx, fcoef[3]);
    if (fent[1]) put(c - 1, fcoef[1]);
    put(c, center);
    if (fent[0]) put(c + 1, fcoef[0]);
    if (fent[2]) put(c + nx, fcoef[2]);
    const int korder[4] = {2, 1, 3, 0};  // corners (x, y), (x+1, y), (x, y+1), (x+1, y+1)
    for (int j = 0; j < 4; ++j)
        if (ok[korder[j]]) put(tIdx[korder[j]], tcoef[korder[j]]);
    P.rowCnt[c] = n;
    P.bRaw[c] = tb;
}
// tilt rows: the four cells around the vertex, each through a full tilted face
__global__ void k2_asm_tilt(Grid2 g, Dev d, Fields2 F, const int* vIdx, Proj P) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = g.nx, ny = g.ny;
    if (v >= (nx + 1) * (ny + 1) || !F.open[v]) return;
    const int x = v % (nx + 1), y = v / (nx + 1);
    const int r = vIdx[v];
    if (r < 0 || x < 1 || y < 1 || x >= nx || y >= ny) {  // boundary tilts are fixed closed
        report(d, DS_MISSING_NODE);
        return;
    }
    double fa[4] = {0, 0, 0, 0}, center = 0, tb = 0, coef[4];
    for (int k = 0; k < 4; ++k) {
        fa[k] += g.hdx * SQRT2;
        double coeff = fa[k] / g.tiltOctDx;
        coef[k] = -coeff;
        center += coeff;
        int sign = k <= 1 ? -1 : 1;
        tb += sign * fa[k] * F.tv[4 * v + k];
    }
    const size_t o = (size_t)r * ROW_W;
    // cells (x-1, y-1), (x, y-1), (x-1, y), (x, y): k = 2, 1, 3, 0; the diagonal last
    const int korder[4] = {2, 1, 3, 0};
    for (int j = 0; j < 4; ++j) {
        int k = korder[j];
        P.padCol[o + j] = ci(g, x + TILT_NB_OCT[k][0], y + TILT_NB_OCT[k][1]);
        P.padVal[o + j] = coef[k];
    }
    P.padCol[o + 4] = r;
    P.padVal[o + 4] = center;
    P.rowCnt[r] = 5;
    P.bRaw[r] = tb;
}
__global__ void k2_zero_rows(Proj P, int rows) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < rows) {
        P.rowCnt[r] = 0;
        P.bRaw[r] = 0;
    }
}

// ------------------------------------------------------------------ pressure correction, dual
// correctVelocityByPressure (include/ast_solver.h:283-324) and constrainVelocity: pressure outside
// the domain is 0 on the y faces; the x walls end closed
__global__ void k2_correct(Grid2 g, Fields2 F, const int* vIdx, const double* p, double dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = g.nx, ny = g.ny;
    const int nv = (nx + 1) * (ny + 1), nmx = (nx + 1) * ny, nmy = nx * (ny + 1);
    if (i < nv && F.open[i]) {
        const int c = vIdx[i];
        const int x = i % (nx + 1), y = i / (nx + 1);
        if (c >= 0 && x >= 1 && y >= 1 && x < nx && y < ny)
            for (int k = 0; k < 4; ++k) {
                int t = ci(g, x + TILT_NB_OCT[k][0], y + TILT_NB_OCT[k][1]);
                F.tv[4 * i + k] += ((k < 2) ? -1 : 1) * dt / g.rho * (p[t] - p[c]) / g.tiltOctDx;
            }
    }
    if (i < nmx) {
        const int x = i % (nx + 1), y = i / (nx + 1);
        double p1 = x < nx ? p[ci(g, x, y)] : 0.0, p0 = x > 0 ? p[ci(g, x - 1, y)] : 0.0;
        double u = F.mx[i] - dt / g.rho * (p1 - p0) / g.dx;
        F.mx[i] = (x == 0 || x == nx) ? 0.0 : u;
    }
    if (i < nmy) {
        const int x = i % nx, y = i / nx;
        double p1 = y < ny ? p[ci(g, x, y)] : 0.0, p0 = y > 0 ? p[ci(g, x, y - 1)] : 0.0;
        F.my[i] -= dt / g.rho * (p1 - p0) / g.dx;
    }
}
// ASTFaceGrid::updateDualGrid with CORRECTION_MAC (include/ast_face_grid.h:69-150): the velocity
// of an open tilt is half the sum of its opposite faces along the two diagonal directions
__global__ void k2_dual(Grid2 g, const uint8_t* open, const double* tv, double* dual) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= (g.nx + 1) * (g.ny + 1) || !open[v]) return;
    const double* u = tv + 4 * v;
    double s02 = u[0] + u[2], s13 = u[1] + u[3];
    double ux = INV_SQRT2 * s02 + INV_SQRT2 * s13;
    double uy = INV_SQRT2 * s02 + -INV_SQRT2 * s13;
    dual[2 * v] = ux * 0.5;
    dual[2 * v + 1] = uy * 0.5;
}

// ------------------------------------------------------------------ advection
// advect (include/ast_solver.h:533-553) in one pass over cells, vertices, x faces and y faces.
// adjustLayout (:471-531) opens a tilt where the back-traced density lies in (0.005, 0.7) and the
// tilt is not fixed; semiLagrangianAST (include/ast_advection.h:18-29) fills the cells and the
// tilts open in the new layout; semiLagrangianASTVector (:31-68) projects the sampled velocity on
// TILT_UNIT_DIR[k % 2] for the tilted faces and takes the face's own component on the MAC faces.
// All reads come from `cur` (and its layout), all writes go to `nxt`.  The density of a vertex in
// the new layout is the value the layout test sampled (same position, same back-trace).
__global__ void k2_advect(Grid2 g, Fields2 cur, Fields2 nxt, const double* dual, const uint8_t* fixedT, int adaptive,
                          double dt) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = g.nx, ny = g.ny;
    const long long nc = (long long)nx * ny, nv = (long long)(nx + 1) * (ny + 1), nmx = (long long)(nx + 1) * ny,
                    nmy = (long long)nx * (ny + 1);
    if (i < nc) {
        const int x = (int)(i % nx), y = (int)(i / nx);
        P2 old = backTrace(g, cur, dual, cellPos(g, x, y), dt);
        nxt.dC[i] = scalarSample(g, cur.dC, cur.dV, cur.open, old);
        nxt.hC[i] = scalarSample(g, cur.hC, cur.hV, cur.open, old);
        return;
    }
    i -= nc;
    if (i < nv) {
        const int x = (int)(i % (nx + 1)), y = (int)(i / (nx + 1));
        const P2 pc = vertPos(g, x, y);
        P2 old{0, 0};
        double dens = 0;
        bool sampled = false, o;
        if (adaptive) {
            old = backTrace(g, cur, dual, pc, dt);
            dens = scalarSample(g, cur.dC, cur.dV, cur.open, old);
            sampled = true;
            o = dens > 0.005 && dens < 0.7 && !fixedT[i];
            nxt.open[i] = o ? 1 : 0;
        } else {
            o = nxt.open[i] != 0;
        }
        if (!o) return;
        if (!sampled) {
            old = backTrace(g, cur, dual, pc, dt);
            dens = scalarSample(g, cur.dC, cur.dV, cur.open, old);
        }
        nxt.dV[i] = dens;
        nxt.hV[i] = scalarSample(g, cur.hC, cur.hV, cur.open, old);
        for (int k = 0; k < 4; ++k) {
            P2 p{pc.x + TILT_OFF[k][0] * g.hdx, pc.y + TILT_OFF[k][1] * g.hdx};
            P2 s = velSample(g, cur, dual, backTrace(g, cur, dual, p, dt));
            const double* up = TILT_OFF[k % 2];  // TILT_UNIT_DIR[k % 2], the same values
            nxt.tv[4 * i + k] = s.x * up[0] + s.y * up[1];
        }
        return;
    }
    i -= nv;
    if (i < nmx) {
        const int x = (int)(i % (nx + 1)), y = (int)(i / (nx + 1));
        nxt.mx[i] = velSample(g, cur, dual, backTrace(g, cur, dual, macPos(g, 0, x, y), dt)).x;
        return;
    }
    i -= nmx;
    if (i < nmy) {
        const int x = (int)(i % nx), y = (int)(i / nx);
        nxt.my[i] = velSample(g, cur, dual, backTrace(g, cur, dual, macPos(g, 1, x, y), dt)).y;
    }
}

// ASTSolver::cfl (include/ast_solver.h:55-70): the lower x and y faces of every cell
__global__ void k2_cfl(Grid2 g, const double* mx, const double* my, unsigned long long* out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    double v = 0;
    if (c < g.nx * g.ny) {
        const int x = c % g.nx, y = c / g.nx;
        double vx = mx[mxi(g, x, y)], vy = my[myi(g, x, y)];
        v = vx * vx + vy * vy;
    }
    for (int o = 16; o > 0; o >>= 1) {
        double w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    if ((threadIdx.x & 31) == 0 && v > 0) atomicMax(out, (unsigned long long)__double_as_longlong(v));
}

// ------------------------------------------------------------------ wavefront MIC(0) sweeps
// The system's cells come first in raster order, so a cell's lower neighbours are the cells below
// and to the left (one anti-diagonal earlier) and its upper ones the cells to the right and above
// and its open corner tilts; a tilt row's lower neighbours are its four cells and it has no upper
// ones.  The forward sweep is therefore one anti-diagonal per step (the cells of a diagonal are
// independent), then the tilt rows in one pass; the backward sweep the tilt rows, then the
// diagonals in reverse.  Every row applies its updates in ascending column order with one fused
// multiply-subtract each and multiplies by its pivot reciprocal last -- the generic sweeps'
// arithmetic (and the oracle's in reduce mode 1), so the result is bit-identical.
//
// One warp per 32 columns, each in a CTA of its own, the CTAs one cluster.  A lane owns a column and
// runs one row behind the lane to its left, so the neighbour below / above is its own previous result
// (a register) and the neighbour to the left / right the adjacent lane's (a shuffle), with no barrier
// anywhere.  Between warps, the boundary lane stores each result into the next CTA's shared memory
// (one slot per row, empty until then: a signalling-NaN bit pattern that no arithmetic produces); the
// reader falls a few steps behind and from then on finds the value waiting.  The per-cell records, the
// residual and the results are stored by the warp's diagonals (Proj::wave), so WAVE_CHUNK steps of
// them are one contiguous piece each, which bulk copies bring into shared memory WAVE_STAGES chunks
// ahead (copies by the lanes of a second warp cost the sweep 30 to 100 cycles a step): the sweeping
// warp has little else to issue than its chain.  An absent neighbour has the entry 0 and the result 0,
// and so have the slots outside the grid: nothing is selected on the way from one step to the next.
//
// What bounds it: the chain, a shuffle and three dependent FP64 operations per diagonal (~280 cycles
// with the records and results of the group; four more operations in the backward sweep where tilts
// are open), over the grid's nx + ny diagonals and ~5 more per warp.  With all columns in one CTA the
// SM's one FP64 pipe (a warp instruction per ~17 cycles, predicated-off ones included) and a block
// barrier per diagonal made a step ~650 cycles.  Per application at 192 x 384 on GB300: 360 -> 172 us;
// whole frames, 213 -> 117 ms there and 7.7 -> 5.9 ms at 45 x 83.
constexpr int WAVE_STAGES = 3;
constexpr int WAVE_MAX_NX = 512;
constexpr int WAVE_THREADS = 256;  // warp 0 sweeps, a thread of warp 1 copies, all do the tilt rows
// one chunk's records: WAVE_CHUNK lines of wRecF or wRecB, of wR or wZ, of wTl and of wTz
constexpr int WAVE_VAL = WAVE_CHUNK * 1024, WAVE_TL = WAVE_VAL + WAVE_CHUNK * 256, WAVE_TZ = WAVE_TL + WAVE_CHUNK * 1024;
constexpr int WAVE_STAGE = WAVE_TZ + WAVE_CHUNK * 1024;
constexpr int WAVE_RING = WAVE_STAGES * WAVE_STAGE;
constexpr int WAVE_PAD = 48;       // edge slots before row 0 and after row ny - 1
constexpr int WAVE_MAX_NY = (224 * 1024 - WAVE_RING) / 8 - 2 * WAVE_PAD;  // rows whose edge fits shared memory

// records of the factorised system for the wavefront kernel (one thread per row)
__global__ void k2_wave_gather(Proj P, const int* vIdx) {
    const int nx = P.wnx, ny = P.wny, nc = nx * ny;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= *P.nDof) return;
    const int q0 = P.rowPtr[r], q1 = P.rowPtr[r + 1];
    if (r >= nc) {  // tilt row: its cells (all columns below r), ascending
        const int t = r - nc;
        int k = 0;
        for (int q = q0; q < q1 && k < 4; ++q) {
            int col = P.col[q];
            if (col >= r) break;
            P.wTc[4 * t + k] = col;
            P.wTv[4 * t + k] = P.Lv[P.tpos[q]];
            ++k;
        }
        for (; k < 4; ++k) {  // an interior tilt always has four cells
            P.wTc[4 * t + k] = -1;
            P.wTv[4 * t + k] = 0;
        }
        return;
    }
    const int x = r % nx, y = r / nx, j = wave_slot(x, y, ny), line = j >> 5, lane = j & 31;
    const int corner[4] = {vIdx[x + y * (nx + 1)], vIdx[x + 1 + y * (nx + 1)], vIdx[x + (y + 1) * (nx + 1)],
                           vIdx[x + 1 + (y + 1) * (nx + 1)]};
    double lb = 0, ll = 0, lr = 0, la = 0;
    double tl[4] = {0, 0, 0, 0};
    bool open = false;
    for (int q = q0; q < q1; ++q) {
        const int col = P.col[q];
        if (col == r - nx) lb = P.Lv[P.tpos[q]];
        else if (col == r - 1) ll = P.Lv[P.tpos[q]];
        else if (col == r + 1) lr = P.Lv[q];
        else if (col == r + nx) la = P.Lv[q];
        else if (col >= nc) {
            for (int k = 0; k < 4; ++k)
                if (corner[k] == col) {
                    tl[k] = P.Lv[q];
                    open = true;
                }
        }
    }
    const double inv = P.invdiag[r];
    P.wRecF[line * 64 + lane] = make_double2(lb, ll);
    P.wRecF[line * 64 + 32 + lane] = make_double2(inv, 0);
    P.wRecB[line * 64 + lane] = make_double2(lr, la);
    P.wRecB[line * 64 + 32 + lane] = make_double2(inv, __longlong_as_double(open));
    for (int k = 0; k < 4; ++k) {
        P.wTl[line * 128 + k * 32 + lane] = tl[k];
        P.wTz[line * 128 + k * 32 + lane] = 0;
    }
    if (open) P.wTf[line / WAVE_CHUNK] = 1;
}

constexpr unsigned long long WAVE_EMPTY = 0x7FF4DEADBEEF0001ull;
constexpr long long WAVE_SPIN_LIMIT = 1LL << 22;
__device__ __forceinline__ double2 wave_ld2(uint32_t a) {
    double2 v;
    asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double wave_ld1(uint32_t a) {
    double v;
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
// Results handed from warp to warp stand in the reader's shared memory or, for grids too tall for that
// (TALL), in global memory; A is the type of their byte addresses, and its width says which.  The reader
// is behind by then: a step is no slower (ms per iteration, GB300: 100 x 20,000 9.1 and, by the generic
// sweeps, 125; 33 x 19,000 9.5 and 102; one warp's 2 x 25,400, which hands nothing on, 9.9 and 13.8).
__device__ __forceinline__ double2 wave_ld2(unsigned long long a) {
    double2 v;
    asm volatile("ld.volatile.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(a) : "memory");
    return v;
}
// a step's result: into wZ where the row is in the grid, into the neighbour's edge from the boundary lane
__device__ __forceinline__ void wave_put(double* out, uint32_t peer, double v, bool on, bool writer) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %3, 0;\n setp.ne.b32 q, %4, 0;\n"
        " @q st.shared::cluster.f64 [%1], %2;\n @p st.global.f64 [%0], %2;\n}" ::"l"(out),
        "r"(peer), "d"(v), "r"((int)on), "r"((int)writer)
        : "memory");
}
__device__ __forceinline__ void wave_put(double* out, unsigned long long peer, double v, bool on, bool writer) {
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %3, 0;\n setp.ne.b32 q, %4, 0;\n"
        " @q st.volatile.global.f64 [%1], %2;\n @p st.global.f64 [%0], %2;\n}" ::"l"(out),
        "l"(peer), "d"(v), "r"((int)on), "r"((int)writer)
        : "memory");
}
__device__ __forceinline__ bool wave_empty(double v) { return __double2hiint(v) == (int)(WAVE_EMPTY >> 32); }
// waits for the phase of `parity`; false past the limit (status), or, given a status, once any wait
// has given up
__device__ __forceinline__ bool wave_wait(uint32_t bar, int parity, int* status) {
    for (long long it = 1; it <= WAVE_SPIN_LIMIT; ++it) {
        int ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.s32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
        if (status && (it & 255) == 0 && *(volatile int*)status != 0) return false;
    }
    if (status) atomicCAS(status, 0, DS_WAIT_TIMEOUT);
    return false;
}
// one warp's columns
struct WaveWarp {
    uint32_t ring, bars;       // records; full[WAVE_STAGES] then freed[WAVE_STAGES]
    int x, line0, chunks, g0;  // this lane's column; the warp's first line; its chunks; chunks of earlier sweeps
};
// the copying thread: the chunks of a sweep in its order, then their completion (nothing is in flight
// when it returns, also when the sweep gave up)
template <bool FWD>
__device__ __forceinline__ void wave_copy(const Proj& P, const WaveWarp& W) {
    int issued = 0;
    for (int c = 0; c < W.chunks; ++c, ++issued) {
        const int g = W.g0 + c, s = g % WAVE_STAGES;
        if (g >= WAVE_STAGES && !wave_wait(W.bars + 8 * (WAVE_STAGES + s), (g / WAVE_STAGES - 1) & 1, P.wStatus)) break;
        const long long line = W.line0 + (FWD ? c : W.chunks - 1 - c) * WAVE_CHUNK;
        const bool tilts = !FWD && P.wTf[line / WAVE_CHUNK] != 0;
        const uint32_t dst = W.ring + s * WAVE_STAGE, bar = W.bars + 8 * s;
        auto bulk = [&](uint32_t to, const void* src, int bytes) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(src),
                         "r"(bytes), "r"(bar)
                         : "memory");
        };
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(tilts ? WAVE_STAGE : WAVE_TL) : "memory");
        bulk(dst, (FWD ? P.wRecF : P.wRecB) + line * 64, WAVE_CHUNK * 1024);
        bulk(dst + WAVE_VAL, (FWD ? P.wR : P.wZ) + line * 32, WAVE_CHUNK * 256);
        if (tilts) {
            bulk(dst + WAVE_TL, P.wTl + line * 128, WAVE_CHUNK * 1024);
            bulk(dst + WAVE_TZ, P.wTz + line * 128, WAVE_CHUNK * 1024);
        }
    }
    for (int c = issued > WAVE_STAGES ? issued - WAVE_STAGES : 0; c < issued; ++c) {
        const int g = W.g0 + c;
        wave_wait(W.bars + 8 * (g % WAVE_STAGES), (g / WAVE_STAGES) & 1, nullptr);
    }
}

// One sweep over the warp's lines, upwards (forward) or downwards (backward).  The boundary lane (0
// forward, 31 backward) takes its neighbour's results from `edge` (by row; the slots outside the
// grid hold 0: no step checks the range; a warp that is not linked to such a neighbour reads one pair of
// zeros all the way), the opposite lane stores its own into `peer` (0: none).  The warp issues in order and pays
// 20 to 30 cycles for each load or store among a step's FP64 operations, so these stand together:
// once per WAVE_GROUP steps, the next group's records and edge values and this group's results.
constexpr int WAVE_GROUP = 2;
struct WaveGroup {
    double2 l[WAVE_GROUP], iv[WAVE_GROUP];
    double v[WAVE_GROUP], edge[WAVE_GROUP];
};
template <bool FWD, typename A>
__device__ __forceinline__ void wave_sweep(const Proj& P, const WaveWarp& W, A edge, A peer, bool linked) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, sd = FWD ? 1 : -1;
    const unsigned bound = W.x < P.wnx ? P.wny : 0;
    const bool first = lane == (FWD ? 0 : 31), writer = peer != 0 && lane == (FWD ? 31 : 0);
    const int start = FWD ? 0 : W.chunks * WAVE_CHUNK - 1;  // the sweep's first line
    int y = start - lane;                                   // this lane's row
    A ea = edge + (A)(linked ? 8 * (start - (FWD ? 0 : 31)) : 0);  // the boundary lane's row
    const int ed = linked ? 8 * WAVE_GROUP * sd : 0;
    A pa = peer + (A)(8 * y);
    double* out = P.wZ + (W.line0 + start) * 32LL + lane;
    double prev = 0;  // this column's last result
    constexpr int G = WAVE_GROUP;
    WaveGroup cur, nxt;
    auto loadEdge = [&](WaveGroup& q) {
#pragma unroll
        for (int k = 0; k + 1 < G; k += 2) {
            const double2 a = wave_ld2(FWD ? ea + 8 * k : ea - 8 - 8 * k);
            q.edge[k] = FWD ? a.x : a.y;
            q.edge[k + 1] = FWD ? a.y : a.x;
        }
    };
    auto load = [&](WaveGroup& q, uint32_t stage, int h) {
#pragma unroll
        for (int k = 0; k < G; ++k) {
            const int i = FWD ? h * G + k : WAVE_CHUNK - 1 - h * G - k;
            q.l[k] = wave_ld2(stage + i * 1024 + lane * 16);
            q.iv[k] = wave_ld2(stage + i * 1024 + 512 + lane * 16);
            q.v[k] = wave_ld1(stage + WAVE_VAL + i * 256 + lane * 8);
        }
    };
    auto empty = [&](const WaveGroup& q) {  // the same slots for all lanes
        bool e = false;
#pragma unroll
        for (int k = 0; k < G; ++k) e = e || wave_empty(q.edge[k]);
        return e;
    };
    auto full = [&](int g) {
        wave_wait(W.bars + 8 * (g % WAVE_STAGES), (g / WAVE_STAGES) & 1, P.wStatus);
        __syncwarp();
        return W.ring + (uint32_t)(g % WAVE_STAGES) * WAVE_STAGE;
    };
    uint32_t stage = full(W.g0);
    load(nxt, stage, 0);
    loadEdge(nxt);
#pragma unroll 1
    for (int c = 0; c < W.chunks; ++c) {
        const int g = W.g0 + c;
        uint32_t next = stage;
#pragma unroll
        for (int h = 0; h < WAVE_CHUNK / G; ++h) {
            for (long long it = 1; empty(nxt); ++it) {
                loadEdge(nxt);
                if ((it & 255) == 0) {
                    if (it > WAVE_SPIN_LIMIT) atomicCAS(P.wStatus, 0, DS_WAIT_TIMEOUT);
                    if (*(volatile int*)P.wStatus != 0)
                        for (int k = 0; k < G; ++k) nxt.edge[k] = 0;
                }
            }
            __syncwarp();
            cur = nxt;
            ea += (A)ed;
            if (h + 1 < WAVE_CHUNK / G) {
                load(nxt, stage, h + 1);
            } else if (c + 1 < W.chunks) {
                next = full(g + 1);
                load(nxt, next, 0);
            }
            loadEdge(nxt);
            double res[G];
#pragma unroll
            for (int k = 0; k < G; ++k) {
                // forward: below (own), then left; backward: right, then above (own), then the corner tilts
                double side = FWD ? __shfl_up_sync(FULL, prev, 1) : __shfl_down_sync(FULL, prev, 1);
                double acc = FWD ? fma(-cur.l[k].x, prev, cur.v[k]) : cur.v[k];
                if (first) side = cur.edge[k];
                acc = fma(FWD ? -cur.l[k].y : -cur.l[k].x, side, acc);
                if (!FWD) acc = fma(-cur.l[k].y, prev, acc);
                // the tilts' entries and results (zero where closed); the forward records have none,
                // but the branch keeps the group's loads and stores out of the chain there too
                // (without it 320 cycles a step instead of 280)
                const int open = __any_sync(FULL, __double2loint(cur.iv[k].y)) ? 4 : 0;
                const uint32_t tl = stage + WAVE_TL + (WAVE_CHUNK - 1 - h * G - k) * 1024 + lane * 8;
#pragma unroll 1
                for (int q = 0; q < open; ++q) acc = fma(-wave_ld1(tl + q * 256), wave_ld1(tl + q * 256 + (WAVE_TZ - WAVE_TL)), acc);
                res[k] = prev = acc * cur.iv[k].x;
            }
#pragma unroll
            for (int k = 0; k < G; ++k) wave_put(out + sd * 32 * k, pa + (A)(8 * sd * k), res[k], (unsigned)(y + sd * k) < bound, writer);
            out += sd * 32 * G;
            pa += (A)(8 * sd * G);
            y += sd * G;
        }
        __syncwarp();
        if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(W.bars + 8 * (WAVE_STAGES + g % WAVE_STAGES)) : "memory");
        stage = next;
    }
}
// z: the tilt rows' results; the cells' stay in wZ
template <bool TALL>
__global__ void __launch_bounds__(WAVE_THREADS, 1) k2_precond_wave(Proj P, const double* r, double* z) {
    extern __shared__ __align__(16) unsigned char wave_smem[];
    __shared__ __align__(8) unsigned long long bars[2 * WAVE_STAGES];
    cg::cluster_group cl = cg::this_cluster();
    if (*P.done) return;
    const int nx = P.wnx, ny = P.wny, nc = nx * ny, n = *P.nDof;
    const int rank = cl.block_rank(), nb = cl.num_blocks(), x0 = 32 * rank;
    typedef typename std::conditional<TALL, unsigned long long, uint32_t>::type A;
    const int rows = nb > 1 ? ny : 0, stride = (rows + 2 * WAVE_PAD + 1) & ~1;  // of an edge
    double* e = TALL ? P.wEdge + (size_t)rank * stride : reinterpret_cast<double*>(wave_smem + WAVE_RING);
    WaveWarp W;
    W.ring = (uint32_t)__cvta_generic_to_shared(wave_smem);
    W.bars = (uint32_t)__cvta_generic_to_shared(bars);
    W.x = x0 + (threadIdx.x & 31);
    W.line0 = rank * wave_lines(ny);
    W.chunks = (ny + min(31, nx - 1 - x0) + WAVE_CHUNK - 1) / WAVE_CHUNK;  // up to the last line with a cell
    W.g0 = 0;
    A edge;  // row 0
    if (TALL) edge = (A)(uintptr_t)(e + WAVE_PAD);
    else edge = (A)(W.ring + WAVE_RING + 8 * WAVE_PAD);
    auto peer = [&](int q, A mine) {
        if (q < 0 || q >= nb) return (A)0;
        if (TALL) return mine + (A)(8LL * (q - rank) * stride);
        uint32_t m = 0;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"((uint32_t)mine), "r"(q));
        return (A)m;
    };
    auto clear = [&](bool neighbour, int row0) {  // row 0 at slot row0
        for (int i = threadIdx.x; i < stride; i += blockDim.x)
            e[i] = neighbour && i >= row0 && i < rows + row0 ? __longlong_as_double((long long)WAVE_EMPTY) : 0.0;
    };
    clear(rank > 0, WAVE_PAD);
    if (threadIdx.x == 32) {
        for (int i = 0; i < 2 * WAVE_STAGES; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(W.bars + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cl.sync();  // every CTA is running and its edge is empty
    if (threadIdx.x < 32) wave_sweep<true, A>(P, W, edge, peer(rank + 1, edge), rank > 0);
    else if (threadIdx.x == 32) wave_copy<true>(P, W);
    __syncwarp();
    __threadfence();
    cl.sync();
    clear(rank + 1 < nb, WAVE_PAD + 1);
    // (rows one slot on: a group's two rows, read as one aligned pair, then start at an odd row)
    // tilt rows: forward (their four cells), then their backward step (no upper entries); the result
    // also goes to the four cells' records for the backward sweep
    for (int tr = nc + rank * blockDim.x + threadIdx.x; tr < n; tr += nb * blockDim.x) {
        const int i = tr - nc;
        double acc = r[tr];
        int slot[4];
        for (int k = 0; k < 4; ++k) {
            const int c = P.wTc[4 * i + k];
            slot[k] = c >= 0 ? wave_slot(c % nx, c / nx, ny) : -1;
            if (c >= 0) acc = fma(-P.wTv[4 * i + k], __ldcg(P.wZ + slot[k]), acc);
        }
        const double inv = P.invdiag[tr];
        acc = acc * inv;
        acc = acc * inv;
        z[tr] = acc;
        for (int k = 0; k < 4; ++k)  // the tilt is corner 3 - k of its k-th cell
            if (slot[k] >= 0) P.wTz[(slot[k] >> 5) * 128 + (3 - k) * 32 + (slot[k] & 31)] = acc;
    }
    __threadfence();
    asm volatile("fence.proxy.async;" ::: "memory");  // wZ and wTz are read by bulk copies
    cl.sync();
    W.g0 = W.chunks;
    if (threadIdx.x < 32) wave_sweep<false, A>(P, W, edge + 8, peer(rank - 1, edge + 8), rank + 1 < nb);
    else if (threadIdx.x == 32) {
        asm volatile("fence.proxy.async;" ::: "memory");
        wave_copy<false>(P, W);
    }
    __syncwarp();
    cl.sync();  // no CTA leaves while a neighbour may still store into its edge
}

}  // namespace g2

using namespace g2;
void launch2_source(const Grid2& g, const Fields2& F, cudaStream_t st) {
    long long n = (long long)(g.nx + 1) * (g.ny + 1);
    ASTG_LAUNCH(k2_source<<<nblk2(n), TB2, 0, st>>>(g, F));
}
void launch2_force(const Grid2& g, const Fields2& F, double dt, cudaStream_t st) {
    long long n = (long long)(g.nx + 1) * (g.ny + 1);
    ASTG_LAUNCH(k2_force<<<nblk2(n), TB2, 0, st>>>(g, F, dt));
}
void launch2_numbering(const Grid2& g, const Fields2& F, int* cnt, int* vIdx, int* bsum, int* total, int* nDof,
                       cudaStream_t st) {
    long long nv = (long long)(g.nx + 1) * (g.ny + 1);
    ASTG_LAUNCH(k2_count<<<nblk2(nv), TB2, 0, st>>>(g, F.open, cnt));
    launch_exclusive_scan(cnt, vIdx, bsum, total, nv, st);
    // vIdx holds the scan; k2_assign reads it through `base` before overwriting the same entry
    ASTG_LAUNCH(k2_assign<<<nblk2(nv), TB2, 0, st>>>(g, F.open, vIdx, total, vIdx, nDof));
}
void launch2_assemble(const Grid2& g, const Dev& d, const Fields2& F, const int* vIdx, Proj& P, double dt,
                      cudaStream_t st) {
    const long long nc = (long long)g.nx * g.ny, nv = (long long)(g.nx + 1) * (g.ny + 1);
    const int rows = (int)(nc + nv);
    ASTG_LAUNCH(k2_zero_rows<<<nblk2(rows), TB2, 0, st>>>(P, rows));
    ASTG_LAUNCH(k2_asm_cell<<<nblk2(nc), TB2, 0, st>>>(g, d, F, vIdx, P));
    ASTG_LAUNCH(k2_asm_tilt<<<nblk2(nv), TB2, 0, st>>>(g, d, F, vIdx, P));
    launch_rows_to_csr(d, P, rows, g.rho / dt, st);
}
void launch2_correct(const Grid2& g, const Fields2& F, const int* vIdx, const double* p, double dt, cudaStream_t st) {
    const long long n = (long long)(g.nx + 1) * (g.ny + 1);
    ASTG_LAUNCH(k2_correct<<<nblk2(n), TB2, 0, st>>>(g, F, vIdx, p, dt));
}
void launch2_dual(const Grid2& g, const Fields2& F, double* dual, cudaStream_t st) {
    const long long n = (long long)(g.nx + 1) * (g.ny + 1);
    ASTG_LAUNCH(k2_dual<<<nblk2(n), TB2, 0, st>>>(g, F.open, F.tv, dual));
}
void launch2_advect(const Grid2& g, const Fields2& cur, const Fields2& nxt, const double* dual, const uint8_t* fixedT,
                    bool adaptive, double dt, cudaStream_t st) {
    const long long n = (long long)g.nx * g.ny + (long long)(g.nx + 1) * (g.ny + 1) + (long long)(g.nx + 1) * g.ny +
                        (long long)g.nx * (g.ny + 1);
    ASTG_LAUNCH(k2_advect<<<nblk2(n), TB2, 0, st>>>(g, cur, nxt, dual, fixedT, adaptive ? 1 : 0, dt));
}
void launch2_cfl(const Grid2& g, const Fields2& F, unsigned long long* out, cudaStream_t st) {
    cudaMemsetAsync(out, 0, sizeof(unsigned long long), st);
    ASTG_LAUNCH(k2_cfl<<<nblk2((long long)g.nx * g.ny), TB2, 0, st>>>(g, F.mx, F.my, out));
}

void launch2_wave_gather(const Proj& P, const int* vIdx, int rows, cudaStream_t st) {
    cudaMemsetAsync(P.wTf, 0, sizeof(int) * (wave_slots(P.wnx, P.wny) / (32 * WAVE_CHUNK)), st);
    ASTG_LAUNCH(k2_wave_gather<<<nblk2(rows), TB2, 0, st>>>(P, vIdx));
}
static bool wave_tall(int nx, int ny) { return nx > 32 && ny > WAVE_MAX_NY; }
long long wave_edge_slots(int nx, int ny) { return wave_tall(nx, ny) ? (nx + 31LL) / 32 * ((ny + 2 * WAVE_PAD + 1) & ~1) : 0; }
static size_t wave_smem_bytes(int nx, int ny) {
    if (wave_tall(nx, ny)) return WAVE_RING;
    return (size_t)WAVE_RING + 8 * (size_t)(((nx > 32 ? ny : 0) + 2 * WAVE_PAD + 1) & ~1);
}
static void wave_config(int nx, int ny, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {
    const int ctas = (nx + 31) / 32;
    cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(WAVE_THREADS);
    cfg.dynamicSmemBytes = wave_smem_bytes(nx, ny);
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}
void launch_precond_wave(const Proj& P, const double* r, double* z, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    wave_config(P.wnx, P.wny, st, cfg, at);
    count_launch();
    note_launch(cudaLaunchKernelEx(&cfg, P.wEdge ? k2_precond_wave<true> : k2_precond_wave<false>, P, r, z));
}
// The wavefront kernel takes up to WAVE_MAX_NX columns (16 CTAs of 32) and any height; its slots use
// 32-bit indices.  Wider grids take the generic sweeps.  Call with the device current.
bool wave_supported(int nx, int ny) {
    if (nx < 2 || nx > WAVE_MAX_NX || wave_slots(nx, ny) * 4 >= (1LL << 31)) return false;
    const void* kern = wave_tall(nx, ny) ? (const void*)k2_precond_wave<true> : (const void*)k2_precond_wave<false>;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    wave_config(nx, ny, nullptr, cfg, at);
    int nc = 0;
    const bool ok =
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wave_smem_bytes(64, WAVE_MAX_NY)) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) == cudaSuccess && nc > 0;
    if (!ok) cudaGetLastError();
    return ok;
}

}  // namespace astg
