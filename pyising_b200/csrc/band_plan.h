// The band height of int8 half-sweeps: host arithmetic only, no CUDA.
#pragma once

namespace ising {

// Default band height: the longest of 16, 8, 4 rows whose slots still make enough waves of resident
// threads (4 blocks of 256 per SM at 64 registers), else 2 (one wave) or 1.  Enough is 5/3 waves, for
// 3D bands of 8 and 4 rows three: with one to two waves most of the second one is empty, and a 3D
// band reuses less (two of a row's five opposite-colour rows are other planes').  Rows of one chunk
// put every lane of a warp in a band of its own, whose rows share no cache lines with the next
// lane's: bands of at most four rows, in 3D two.  Over 70 shapes from 264^3 to 900x100x1000 and 4200^2
// to 16000^2 this is 10% (3D) and 3% (2D) faster than the longest band of one wave and nowhere more
// than 1.3% slower.  Measured on one B200, flips/ns, one wave -> this: 2D 7000x7000 950 -> 1019, 9000x9000
// 933 -> 1063, 2000000x32 749 -> 1065; 3D heat bath 300x300x304 681 -> 765, 448^3 689 -> 1002,
// 1000x1000x24 502 -> 584, 2000x2000x32 504 -> 915.
inline int int8_default_band(long long rows, int ly, int cpr, int sm_count)
{
    const long long resident = 1024LL * sm_count, planes = rows / ly;
    auto slots = [&](int b) { return planes * ((ly + b - 1) / b) * cpr; };
    auto enough = [&](int b) {
        return 3 * slots(b) >= (planes > 1 && b < 16 ? 9 : 5) * resident;
    };
    int b = cpr > 1 ? 16 : (planes > 1 ? 2 : 4);
    while (b > 2 && !enough(b)) b >>= 1;
    while (b > 1 && slots(b) < resident) b >>= 1;
    return b;
}

// Longest band of batched half-sweeps for a lattice of rows of `cpr` chunks, whatever the class has to
// spare: in rows of one chunk (see above) four rows, in 3D two, and in 3D bands of 8 rows pay from 16
// chunks on only.  Measured on one B200, us, bands of 8 -> this: 3D heat bath 6 x 1000x1000x24 8006 ->
// 4509, 4 x 2000x2000x32 4000 -> 2698, 4 x 300x300x304 3235 -> 2817, 2 x 400x400x416 3058 -> 2687; 2D 4 x
// 2000000x32 2880 -> 2115; and bands of 4 -> 8: 2 x 512^3 2333 -> 2239, 4 x 100x1000x1000 3859 -> 3720.
inline int int8_band_limit(int ndim, int cpr)
{
    if (cpr == 1) return ndim == 3 ? 2 : 4;
    return ndim == 3 && cpr < 16 ? 4 : 64;
}

}  // namespace ising
