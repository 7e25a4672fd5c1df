// Reads of the state that plan_pauli_sum asks for: prints "qubits precision kind count passes left_out parts"
// for lists of random Z strings, alone and beside flips.
#include <cstdio>
#include <random>
#include <vector>

#include "qm_internal.h"

int main() {
    std::mt19937 rng(7);
    auto list = [&](int qubits, int count, bool flips) {
        std::vector<qm_pauli_term> terms((size_t)count);
        for (int i = 0; i < count; ++i) {
            qm_pauli_term& t = terms[(size_t)i];
            t = qm_pauli_term{};
            t.sign_mask = 1u + rng() % ((1u << qubits) - 1u);
            t.coefficient = 1.0;
            if (flips && i % 2) {
                t.flip_mask = 3u << (i % (qubits - 1));
                t.sign_mask &= ~t.flip_mask;
            }
        }
        return terms;
    };
    for (int qubits : {17, 20, 24, 28})
        for (int precision : {QM_FP64, QM_FP32})
            for (bool flips : {false, true})
                for (int count : {64, 256, 1000}) {
                    const auto terms = list(qubits, count, flips);
                    qm::PauliSumPlan plan;
                    qm::plan_pauli_sum(qubits, precision, terms.data(), count, 148, plan);
                    std::printf("%d %d %s %d %d %zu %d\n", qubits, precision, flips ? "mixed" : "diagonal", count,
                                plan.passes, plan.wide.size(), plan.parts);
                }
}
