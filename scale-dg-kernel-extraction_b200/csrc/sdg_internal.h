// Internal helpers shared by the host set-up and the GPU core.
#pragma once

#include <string>
#include <vector>

namespace sdg {

// Records a formatted message as the calling thread's last error and
// returns `code`.
int fail(int code, const char* fmt, ...);
const std::string& last_error();

// Reference faces 1..6 as 0..5: normal axis (0 x, 1 y, 2 z), sign and the
// opposite face (mod_mesh.f90:266-276, 420-480).
extern const int kFaceAxis[6];
extern const double kFaceSign[6];
extern const int kOppFace[6];

// Fmask(fp+1, f+1) - 1: the 0-based element node of face node fp on face f.
int face_node(int Nq, int f, int fp);

// Relative tolerance of the factored lift: the largest tangential spread
// of a Lift_mat column, relative to max|Lift_mat|, that the fast kernels
// accept.  The reference's operator files spread by at most 2.4e-14
// (p = 15) and 3.4e-15 (p = 7).
constexpr double kLiftFactorTol = 1e-13;

// Tensor-product factorisation of Lift_mat(Np, 6).  On a hexahedron with
// tensor-product nodes, Lift(i,j,k,f) depends only on the node index
// along face f's normal; `expanded` receives the table rebuilt from the
// first tangential row of each face (entry (i,j,k,f) = Lift at normal
// index n, tangential indices 0) and `lift_z` the factors l_f(n) of the faces
// -z, +z, -x, +x, -y, +y, Nq each.  Returns false (and
// leaves the outputs empty) when some entry differs from its factor by
// more than kLiftFactorTol * max|Lift_mat|.
bool lift_factor(const double* Lift, int Nq, std::vector<double>* expanded,
                 std::vector<double>* lift_z);

// Steps of the longer step graph of a handle, and whether a call of nsteps steps
// captures it, given the steps of this dt asked for so far (this call's included).
// Capturing it costs 0.13 to 0.2 ms and gives 0 to 2 us a step, so a program that
// changes dt with each call of a few dozen steps must not pay for it each time: 24
// steps of a new dt took 500 us with it at 4^3, p = 3, 370 without, and 8^3, p = 5
// gained nothing in a first call of 100 steps.
constexpr int kGraphSteps = 8;
constexpr long long kGraphStepsFrom = 128;
constexpr bool step_graph_pays(long long asked, int nsteps) {
  return nsteps >= kGraphSteps && asked >= kGraphStepsFrom;
}

}  // namespace sdg
