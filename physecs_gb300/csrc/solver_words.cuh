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

// ---- colouring: a contact's claim on a body.  The lowest claim wins: by colour (7 bits),
// then a hash of 16 bits, then the contact's index within its scene, in 32 bits, by which it
// knows its claim again.  No claim: all ones.
PSX_WORD unsigned long long claim_word(int colour, unsigned hash, int contact) {
    return (unsigned long long)colour << 48 | (unsigned long long)(hash & 0xffffu) << 32 | (unsigned)contact;
}
PSX_WORD bool claim_of(unsigned long long word, int contact) { return (unsigned)word == (unsigned)contact; }
PSX_WORD int claim_colour(unsigned long long word) { return (int)(word >> 48); }

// ---- point slots of a contact in the solve order: its first slot (29 bits) and the step
// between its points (1 to 8).  A contact has at most four points, so the slots of up to
// kMaxContacts contacts stay in their field; a world has room for no more (a frame with more
// reports the manifold capacity).
constexpr long long kMaxContacts = 1ll << 27;
PSX_WORD int contact_room(int per_collider, int colliders) {
    const long long n = (long long)per_collider * colliders;
    return (int)(n < 1024 ? 1024 : n < kMaxContacts ? n : kMaxContacts);
}
PSX_WORD int slot_word(int first, int step) { return (int)((unsigned)first | (unsigned)(step - 1) << 29); }
PSX_WORD int slot_first(int word) { return (int)((unsigned)word & 0x1fffffffu); }
PSX_WORD int slot_step(int word) { return (int)((unsigned)word >> 29) + 1; }

}  // namespace psx
