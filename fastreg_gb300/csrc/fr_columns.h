// fr_columns.h -- how the threads of the adjoint's column kernels lie over a volume.
//
// Header-only, plain C++ outside nvcc: fr_adjoint.cu includes it, and a CPU test compiles it on its own.
#pragma once

#ifdef __CUDACC__
#define FR_COLUMNS_FN __device__ __forceinline__
#else
#define FR_COLUMNS_FN inline
#endif

namespace frg {

// A thread owns a column of `depth` slices.  A block's 256 columns are one of
//   - a tile of 32 x 8, where that leaves as few threads idle as the next (fr_warp_adjoint on 160x192x160:
//     57.4 us, 58.0 flat; on 128^3 33.5 and 35.1),
//   - flat: consecutive voxels of a slice, rows running on, so that only the slice's last block has idle threads
//     (130x150x130 45.5 us, 48.9 in tiles; 33x200x200 25.7 and 33.4; 5x512x512 22.2 and 69.9; a
//     gradient of 97x115x97 at width 11 1.91 ms, 2.04 in tiles),
//   - layered, where a slice is less than half a block: 2^lx by 2^ly columns in several layers of a block
//     (4x4x20000 9.9 us, 36.6 in tiles).  The kernels' loop is not uniform over the block any more then, which
//     takes up to 32 registers more; a warp lies in one layer, as its lanes share their loop.
// On 49 sizes from 40x135x40 to 192x224x192 the rule between the first two is within 4% of the faster.
enum ColumnShape { kTileColumns, kFlatColumns, kLayeredColumns };
struct Columns {
    ColumnShape shape = kFlatColumns;
    int pitch;           // of a row
    int lx = 8, ly = 0;  // a block's columns along x and y (flat: 2^8 in all)
    int nx, ny = 1;      // blocks of a layer along x and y (flat: nx)
    int depth = 1;
    // rows of X voxels `pitch` apart, Y of them
    Columns(int pitch, int X, int Y) : pitch(pitch), nx((pitch * Y + 255) / 256) {
        const int tx = (X + 31) / 32, ty = (Y + 7) / 8;
        if (pitch * Y <= 128) {
            int least = 256;  // the whole slice in the fewest threads, wide before tall
            for (int x = 5; x >= 0; --x)
                for (int y = 7 - x; y >= 5 - x; --y)
                    if ((1 << x) >= X && (1 << y) >= Y && 1 << (x + y) < least) {
                        least = 1 << (x + y);
                        shape = kLayeredColumns;
                        lx = x;
                        ly = y;
                        nx = 1;
                    }
        } else if (100LL * tx * ty <= 102LL * nx) {
            shape = kTileColumns;
            lx = 5;
            ly = 3;
            nx = tx;
            ny = ty;
        }
    }
    int layers() const { return 256 >> (lx + ly); }
    long long blocks(int Z) const {
        const long long n = ((long long)Z + depth - 1) / depth;
        return (long long)nx * ny * ((n + layers() - 1) / layers());
    }
    // the column of thread t of block b: x, y (possibly outside the volume) and its slices z0 .. z1 - 1 (none if
    // z0 >= z1)
    template <int SHAPE>
    FR_COLUMNS_FN void place(int b, int t, int Z, int& x, int& y, int& z0, int& z1) const {
        int layer;
        if (SHAPE == kTileColumns) {
            layer = b / (nx * ny);
            x = b % nx * 32 + (t & 31);
            y = b / nx % ny * 8 + (t >> 5);
        } else if (SHAPE == kFlatColumns) {
            layer = b / nx;
            const int col = (b - layer * nx) * 256 + t;
            y = col / pitch;
            x = col - y * pitch;
        } else {
            x = t & ((1 << lx) - 1);
            y = (t >> lx) & ((1 << ly) - 1);
            layer = b * (256 >> (lx + ly)) + (t >> (lx + ly));
            if (layer > (Z - 1) / depth) {
                z0 = z1 = Z;
                return;
            }
        }
        z0 = layer * depth;
        z1 = Z - z0 > depth ? z0 + depth : Z;
    }
};

}  // namespace frg
