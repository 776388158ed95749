// Clustering steps of ploc.cu, block by block on the CPU (host_block.hpp); the
// kernel's source precedes this text in the same translation unit.
namespace mrb {
namespace {

struct Step {
    uint32_t n;
    std::vector<float> boxes, inner;
    std::vector<uint32_t> sorted, C, Cout, left, right;
    std::vector<unsigned long long> status;
    PlocState state[2];
    uint32_t root = 0, ticket = 0, error = 0;

    explicit Step(uint32_t count)
        : n(count), boxes(6 * count), inner(6 * count), sorted(count), C(count),
          Cout(count, 0xABABABABu), left(count), right(count), status(step_tiles(count), 0ull) {
        uint32_t r = 1;
        for (uint32_t i = 0; i < n; i++) {
            sorted[i] = C[i] = i;
            for (int c = 0; c < 3; c++) {
                r = r * 1664525u + 1013904223u;
                boxes[6 * i + c] = float(r >> 8);
                boxes[6 * i + 3 + c] = float(r >> 8) + 100.0f;
            }
        }
        state[0] = PlocState{n, 0u, 0u};
        state[1] = PlocState{0u, 0u, 0u};
    }
    // One block; give_up >= 0: another block's look-back gives up when this
    // thread has run to its first synchronisation.
    bool block(uint32_t b, int give_up = -1) {
        blockIdx.x = b;
        bool first = true;
        return host_block::run(
            kStepBlock,
            [&] {
                k_ploc_step(C.data(), Cout.data(), PlocIn{n, boxes.data(), sorted.data()},
                            PlocOut{left.data(), right.data(), inner.data(), &root}, &state[0],
                            &state[1], &ticket, &error, status.data());
            },
            [&](uint32_t t) {
                if (first && int(t) == give_up) error = 1u;
                if (int(t) + 1 == kStepBlock) first = false;
            });
    }
};

int failures = 0;
void expect(bool ok, const char* what, int at) {
    if (!ok) {
        std::printf("%s (%d)\n", what, at);
        failures++;
    }
}

void steps() {
    // the emulation itself: a whole step keeps every cluster, merged or not
    Step s(2000);
    for (uint32_t b = 0; b < step_tiles(s.n); b++) expect(s.block(b), "a step's block", int(b));
    const PlocState& next = s.state[1];
    expect(next.m < s.n && next.m + next.base == s.n && next.steps == 1u, "a step", int(next.m));
    for (uint32_t i = 0; i < next.m; i++)
        expect(s.Cout[i] < s.n + next.base && (i == 0 || s.Cout[i] != s.Cout[i - 1]), "cluster",
               int(i));
}

// The give-up word may be set at any moment.  A block acts on one reading of
// it: its threads all take part in the step or all leave.
void give_up_while_a_block_starts() {
    for (int t : {0, 1, 31, 32, 150, kStepBlock - 2}) {
        Step s(2000);
        for (uint32_t b = 0; b < 3; b++) s.block(b);
        expect(s.block(3, t), "threads of one block part ways", t);
        const std::vector<uint32_t> before = s.Cout;
        expect(s.block(4), "a block after the give-up", t);
        expect(s.Cout == before, "a block after the give-up writes", t);
    }
}

// The arrays of a build neither overlap nor run out of the allocation, at
// counts whose byte sizes pass 32 bits too.
void arrays_of_large_builds() {
    for (uint32_t n : {2u, 1000000u, 178956971u, 178956972u, 200000000u, 0x7FFFFFFFu}) {
        const PlocArrays a = ploc_arrays(n);
        const size_t inner = size_t(n) - 1;
        const size_t at[6] = {a.left, a.right, a.inner, a.root, a.scratch, a.bytes};
        const size_t need[5] = {4 * inner, 4 * inner, 24 * inner, 4, 8 * size_t(n)};
        for (int i = 0; i < 5; i++)
            expect(at[i] % 256 == 0 && at[i] + need[i] <= at[i + 1], "an array's room", int(n));
    }
}

}  // namespace
}  // namespace mrb

int main(int, char** argv) {
    if (!std::strcmp(argv[1], "arrays")) {
        mrb::arrays_of_large_builds();
        return mrb::failures ? 1 : 0;
    }
    mrb::steps();
    mrb::give_up_while_a_block_starts();
    return mrb::failures ? 1 : 0;
}
