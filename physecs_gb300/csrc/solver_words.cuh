// solver_words.cuh — the packed words of the solver and the ranges their fields hold.
//
// Plain C++ as well as CUDA, so that a host test can evaluate the packings at the ends of
// their ranges (tests/test_solver_words.py).
#pragma once
#include <cstdint>

#ifndef __CUDACC__
#define PSX_WORD inline
#else
#define PSX_WORD __host__ __device__ __forceinline__
#endif

namespace psx {

// ---- solve_flow: the word beside a body's pseudo velocity counts the joint rows applied to
// it (what the position integration divides by) and the joints whose preSolve is done (what
// the next joint waits for), 16 bits each.  A joint has at most kMaxRowsPerJoint = 8 rows,
// so the row count stays in its half up to 8191 joints on a body; a scene with a body of
// more joints is solved with barriers.
constexpr int kFlowJoints = 8191;
PSX_WORD int flow_pseudo(int rows, int joints) { return (int)((unsigned)rows | (unsigned)joints << 16); }
PSX_WORD int flow_pseudo_rows(int word) { return (int)((unsigned)word & 0xffffu); }
PSX_WORD int flow_pseudo_joints(int word) { return (int)((unsigned)word >> 16); }

// A body's contacts, and its contacts and joints (its solves in an iteration): at most 127
// contacts (one a colour) and kFlowJoints joints.
PSX_WORD int flow_degree(int contacts, int joints) { return (int)((unsigned)contacts | (unsigned)(contacts + joints) << 16); }
PSX_WORD int flow_contacts(int degree) { return (int)((unsigned)degree & 0xffffu); }
PSX_WORD int flow_solves(int degree) { return (int)((unsigned)degree >> 16); }

}  // namespace psx
