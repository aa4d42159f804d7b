// attn_rows_lanes.cuh -- which value columns and keys a lane of attn_rows_kernel takes: plain arithmetic, also compiled for the host, where a test looks at the
// addresses that follow from it.
#pragma once
#ifdef __CUDACC__
#define AR_HD __host__ __device__ __forceinline__
#else
#define AR_HD inline
#endif

#define AR_THREADS 512
#define AR_WARPS (AR_THREADS / 32)
#define AR_COLS 1024                     // value columns of a unit

// value columns of the unit cb, and the floats its rows of sums take (the last unit of several has fewer columns than that)
AR_HD int ar_cols(int dv, int cb) { return dv - cb * AR_COLS < AR_COLS ? dv - cb * AR_COLS : AR_COLS; }
AR_HD int ar_dvp(int dv) { return dv > AR_COLS ? AR_COLS : (dv + 3) & ~3; }

// a warp's part of the values: 128 columns, 8 heads or fewer (HG groups of heads), every kgs-th key from kg on
struct ArLane {
    int kgs, cg, hg, kg, col;
    bool sums, loads;                    // has sums to pass on (all dvp columns) ; reads values: columns behind the row belong to other rows, or to nobody
};
AR_HD ArLane ar_lane(int w, int lane, int dvp, int cols, int HG) {
    ArLane l;
    const int cgs = (dvp + 127) / 128;
    l.kgs = AR_WARPS / (cgs * HG); l.cg = w % cgs; l.hg = w / cgs % HG; l.kg = w / (cgs * HG); l.col = l.cg * 128 + lane * 4;
    l.sums = l.kg < l.kgs && l.col < dvp; l.loads = l.sums && l.col < cols;
    return l;
}
