// Evaluator calls of a separately compiled program that no part of the library makes itself: stack and tensorAccumulateHalves give the
// residues of concat and of tensorAccumulate on the two halves; multSums refuses terms and masks that do not make whole sums.  Returns 0 when
// they do.
#include "HEMMer.hpp"

#include <cstdio>
#include <vector>

int main() {
    const int d = 16; // N = 2^10: two tiles fill the 512 slots
    hb_params prm = {10, 8, 3, 3, 60, 42, 60, 32, 3.2, {1, 2, 3, 4}};
    HELLM::HEMMer *hemmer = HELLM::HEMMer::genHEMMer(/*device*/ 0, prm);
    const HELLM::Evaluator &ev = hemmer->eval();
    std::vector<double> x(d * d, 0.25), y(d * d, -0.5);
    auto residues = [&](const HELLM::Ciphertext &t) {
        int level = 0, polys = 0, batch = 0, sp = 0;
        hb_ct_meta(t.raw(), &level, &polys, &batch, &sp);
        std::vector<uint64_t> r((size_t)batch * polys * (level + 1) * 1024);
        HELLM::check(hemmer->context(), hb_ct_export(hemmer->context(), t.raw(), r.data()));
        return r;
    };
    std::vector<HELLM::Ciphertext> parts;
    for (int k = 0; k < 3; ++k) {
        std::vector<HELLM::Ciphertext> pair;
        pair.push_back(hemmer->encrypt2(x.data(), y.data(), d, d, /*nonce*/ 2 * k + 1).get());
        pair.push_back(hemmer->encrypt2(y.data(), x.data(), d, d, 2 * k + 2).get());
        parts.push_back(ev.concat(pair)); // two members each
    }
    int bad = 0;
    const HELLM::Ciphertext stacked = ev.stack(parts);
    if (stacked.getBatch() != 6 || residues(stacked) != residues(ev.concat(parts))) ++bad;
    HELLM::Ciphertext halves, plain;
    for (int k = 0; k < 2; ++k) { // into an empty accumulator, then into a filled one
        ev.tensorAccumulateHalves(halves, stacked);
        ev.tensorAccumulate(plain, ev.view(stacked, 0, 3), ev.view(stacked, 3, 3));
        if (residues(halves) != residues(plain)) ++bad;
    }
    std::vector<HELLM::Ciphertext> terms;
    for (int k = 0; k < 3; ++k) terms.push_back(ev.view(stacked, k, 1));
    const HELLM::Plaintext mask = ev.encode(HELLM::Message((size_t)512), terms[0].getLevel());
    const std::vector<const HELLM::Plaintext *> three(3, &mask), two(2, &mask);
    const auto refused = [&](const std::vector<HELLM::Ciphertext> &x, const std::vector<const HELLM::Plaintext *> &p, int count) {
        try { ev.multSums(x, p, count); } catch (const std::invalid_argument &) { return true; }
        return false;
    };
    if (refused(terms, three, 3) || refused(terms, three, 1)) ++bad;
    if (!refused(terms, three, 2) || !refused(terms, three, 0) || !refused(terms, three, -1) || !refused(terms, two, 1) || !refused({}, {}, 1)) ++bad;
    delete hemmer;
    std::printf("%d of 5 results differ\n", bad);
    return bad ? 1 : 0;
}
