// check_words.cpp — the solver's packed words (physecs_gb300/csrc/solver_words.cuh) at the
// ends of their fields' ranges (test infrastructure).  Prints the first field that does not
// come back and returns 1.
#include <cstdio>
#include "solver_words.cuh"

using namespace psx;

#define CHECK(cond)                                                                  \
    do {                                                                             \
        if (!(cond)) { std::printf("line %d: %s\n", __LINE__, #cond); return 1; }    \
    } while (0)

static int flow_words() {
    // a body's joints one after another, each applying all the rows a joint may have
    for (int rows_per_joint = 0; rows_per_joint <= 8; ++rows_per_joint) {
        int word = 0;
        for (int done = 0; done < kFlowJoints; ++done) {
            CHECK(flow_pseudo_joints(word) == done);
            CHECK(flow_pseudo_rows(word) == done * rows_per_joint);
            word = flow_pseudo(flow_pseudo_rows(word) + rows_per_joint, done + 1);
        }
        CHECK(flow_pseudo_joints(word) == kFlowJoints && flow_pseudo_rows(word) == kFlowJoints * rows_per_joint);
    }
    const int contacts[] = {0, 1, 126, 127}, joints[] = {0, 1, 255, 256, kFlowJoints};
    for (int c : contacts)
        for (int j : joints) CHECK(flow_contacts(flow_degree(c, j)) == c && flow_solves(flow_degree(c, j)) == c + j);
    return 0;
}

static int claim_words() {
    const int contacts[] = {0, 1, (1 << 24) - 1, 1 << 24, (1 << 24) + 5, (int)kMaxContacts - 1, 0x7fffffff};
    const unsigned hashes[] = {0u, 1u, 0xffffu, 0xabcd1234u};
    for (int k : contacts) {
        CHECK(!claim_of(~0ull, k));
        for (int c = 0; c < 128; ++c)
            for (unsigned h : hashes) {
                const unsigned long long v = claim_word(c, h, k);
                CHECK(v != ~0ull && claim_colour(v) == c);
                for (int other : contacts) CHECK(claim_of(v, other) == (other == k));
                // the lower colour first, then the hash, then the contact
                for (unsigned g : hashes)
                    for (int other : contacts) {
                        if (c) CHECK(claim_word(c - 1, g, other) < v);
                        if ((g & 0xffffu) < (h & 0xffffu)) CHECK(claim_word(c, g, other) < v);
                        if (other < k) CHECK(claim_word(c, h, other) < v);
                    }
            }
    }
    return 0;
}

static int slot_words() {
    const long long firsts[] = {0, 1, (1ll << 28) - 1, 1ll << 28, 4 * kMaxContacts - 4, 4 * kMaxContacts - 1};
    for (long long first : firsts)
        for (int step = 1; step <= 8; ++step) {
            const int w = slot_word((int)first, step);
            CHECK(slot_first(w) == first && slot_step(w) == step);
        }
    CHECK(contact_room(4, 20) == 1024 && contact_room(4, 1000) == 4000 && contact_room(16, 1 << 23) == kMaxContacts);
    CHECK(contact_room(17, 1 << 23) == kMaxContacts && contact_room(0x7fffffff, 1 << 23) == kMaxContacts);
    return 0;
}

int main() { return flow_words() || claim_words() || slot_words(); }
