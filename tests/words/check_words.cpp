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

int main() { return flow_words(); }
