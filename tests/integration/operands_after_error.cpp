// Row sums of ciphertexts at level 0: the mask multiplication inside them has no level left to rescale into and throws.  The caller's
// operands must still be valid handles with the residues they had.  Returns 0 when they are.
#include "HEMMer.hpp"

#include <cstdio>
#include <functional>
#include <vector>

int main() {
    const int d = 16; // N = 2^10: two tiles fill the 512 slots
    hb_params prm = {10, 8, 3, 3, 60, 42, 60, 32, 3.2, {1, 2, 3, 4}};
    HELLM::HEMMer *hemmer = HELLM::HEMMer::genHEMMer(/*device*/ 0, prm);
    std::vector<double> x(d * d, 0.25), y(d * d, -0.5);
    auto residues = [&](const HELLM::CtxtTensor &t) {
        std::vector<uint64_t> r((size_t)2 * 1024);
        HELLM::check(hemmer->context(), hb_ct_export(hemmer->context(), t.get().raw(), r.data()));
        return r;
    };
    const std::function<void(HELLM::CtxtTensor &, HELLM::CtxtTensor &)> calls[] = {
        [&](HELLM::CtxtTensor &a, HELLM::CtxtTensor &b) { hemmer->oneMatRotSumInplace(a, b); },
        [&](HELLM::CtxtTensor &a, HELLM::CtxtTensor &b) { hemmer->trOneMatRotSumInplace(a, b); },
    };
    int bad = 0;
    for (const auto &call : calls)
        for (int level_b : {0, 1}) { // together as one ciphertext, and each on its own
            auto a = hemmer->encrypt2(x.data(), y.data(), d, d, /*nonce*/ 1), b = hemmer->encrypt2(y.data(), x.data(), d, d, 2);
            a.get() = hemmer->eval().levelDown(a.get(), 0);
            b.get() = hemmer->eval().levelDown(b.get(), level_b);
            const auto before = residues(a);
            bool threw = false;
            try { call(a, b); } catch (const std::invalid_argument &) { threw = true; }
            if (!threw || a.get().empty() || b.get().empty() || a.getLevel() != 0 || b.getLevel() != level_b || residues(a) != before) ++bad;
        }
    delete hemmer;
    std::printf("%d of 4 calls lost an operand\n", bad);
    return bad ? 1 : 0;
}
