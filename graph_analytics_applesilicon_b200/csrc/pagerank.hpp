// pagerank.hpp -- the PageRank handle behind gb_pr_* (the role of
// gpu::GpuPageRank, src/metal/pagerank_gpu.hpp:46-127).
#pragma once

#include <map>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "host_copy.hpp"

constexpr uint32_t kGsHubMin = 4096;  // natural-order GS: split vertices with this many in-edges
constexpr uint32_t kGsNatSlices = 8;    // natural-order GS: the main list runs as this many ordered launches

// Iteration control, updated on the device by the last block of every
// iteration kernel: which rank buffer is current, how many iterations ran,
// and the tol-mode stop rule (L1 change, max relative change, stagnation
// guard of src/metal/pagerank_gpu.mm:384-402).  Kernels launched after a stop
// return immediately, so iteration batches can be CUDA-graph replays.
struct GbPrControl {
    int cur;
    int iters;
    int stopped;
    int floorStop;
    int sinceBest;
    int cap;
    unsigned done;  // last-block-done ticket
    int withDelta;
    double best;
    double lastDelta;
    double lastMaxRel;
    double tol;
    double tolRel;
    float dangHi, dangLo;   // dangling rank of the current iterate (float-float)
    double dang64;          // same, double-precision variant
    double sum64;           // in-place variants: sum of the new iterate
    int error;              // a bounded device wait gave up (the run is invalid)
};

// Blocked pull (GB_PR_PULL_BLOCKED): rows in blocks of at most kBlkRowCap
// (their sums in shared memory, one CUDA block per row block), columns in
// parts of kBlkPart vertices (their contributions staged in shared memory by
// TMA, kBlkCStages parts at a time); tile (row block, part) holds that block's
// edges from that part as packed 32-bit words, staged by TMA in chunks of at
// most kBlkChunk 16-byte words, kBlkEStages chunks at a time.  One producer
// warp issues the copies; kBlkConsumerWarps warps add the edges.  Rows with
// kBlkHub or more in-edges are summed apart.
constexpr uint32_t kBlkPart = 8192;
constexpr uint32_t kBlkRowCap = 21504;
constexpr int kBlkCStages = 2;
constexpr int kBlkEStages = 4;
constexpr int kBlkThreads = 1024;
constexpr int kBlkConsumerWarps = kBlkThreads / 32 - 1;
constexpr uint32_t kBlkChunk = kBlkConsumerWarps * 32;  // one 16-byte word per consumer thread
constexpr uint32_t kBlkHub = 4096;  // rows with this many in-edges are summed apart, one block each

// Contributions an adaptive sweep keeps in shared memory, at most (128 KB): more
// leave the L1 too little room for the gathers in flight (Chung-Lu, 233M entries:
// 24K 736 us a sweep, 32K 717, 40K 710, 48K 793, 56K 1,390; none 820).
constexpr uint32_t kPrHotMax = 32u * 1024u;

constexpr size_t kPrGraphs = 64;  // cached graphs of a handle, at most

// A run of the adaptive layout: vertices [v0, vEnd), all with lists of `vecs`
// vectors, handled by groups of 1 << lg lanes.  Lists follow one another from
// vector e0 on; `inter`: in blocks of 32 lists with vector k of the 32 lists
// side by side, so a lane per list reads whole lines.  The run's warp tasks
// (32 >> lg vertices each) are [task0, next run's task0).
struct GbPrRun {
    uint32_t task0, v0, vEnd, e0, vecs, lg, inter, pad;
};

struct gb_pr {
    uint64_t n = 0, mOut = 0, mIn = 0;
    bool hasOut = false, hasIn = false;
    gb::DevBuf<uint32_t> rowOut, colOut, rowIn, colIn, outdeg;
    gb::DevBuf<float> r[2], contrib[2], acc, accLo;
    gb::DevBuf<double> r64[2], contrib64[2];
    gb::DevBuf<GbPrControl> ctl;
    gb::DevBuf<float> partF;       // per-block float partials (2 per block)
    gb::DevBuf<double> partD;      // per-block double partials (2 per block)
    gb::Stream stream;
    gb::EventPair ev;
    std::vector<uint32_t> hostRowIn, hostColIn, hostOutdeg;

    // adaptive pull (pr_layout.cu): vertices relabeled by descending in-degree
    // (new id = rank), lists sorted and padded to whole 16-byte vectors, and a
    // run per padded length, so a list's place follows from its id
    gb::DevBuf<uint4> vecA;          // the lists
    gb::DevBuf<uint32_t> outdegA;    // by new id
    gb::DevBuf<uint32_t> posA;       // by new id: place of its contribution (with hotA > 0)
    uint32_t hotA = 0;               // contributions worth a copy in shared memory; theirs are places [0, hotA)
    gb::DevBuf<uint32_t> permADev;   // old id -> new id
    gb::DevBuf<GbPrRun> runsA;
    uint32_t nRuns = 0, nRunTasks = 0;
    gb::DevBuf<uint4> hubChunks;     // split lists: (vertex, first vector, end vector, hub index) per chunk
    gb::DevBuf<uint32_t> hubFirst;   // per hub: first chunk | chunk count
    gb::DevBuf<unsigned> hubDone;    // per hub: chunks finished (reset by the last)
    gb::DevBuf<float> hubPart;       // per chunk: its sum (float-float)
    uint32_t nHubs = 0, nChunks = 0;
    // scalar and vector pulls: lanes per list (log2) and the split lists
    struct PrSplit {
        gb::DevBuf<uint4> chunks;  // (vertex, start, end, hub index)
        gb::DevBuf<uint32_t> first;
        gb::DevBuf<unsigned> done;
        gb::DevBuf<float> part;
        uint32_t nChunks = 0, lg = 0, splitMin = 0;
        bool ready = false;
    } split[2];
    uint32_t binSmall = 0, binLarge = 0;
    bool binsReady = false;
    // Gauss-Seidel natural order: vertices of in-degree >= kGsHubMin are split
    // into warp chunks (natural ids) and swept first, in place
    gb::DevBuf<uint4> gsHubChunks;
    gb::DevBuf<uint32_t> gsHubFirst;
    gb::DevBuf<unsigned> gsHubDone;
    gb::DevBuf<float> gsHubPart;
    uint32_t gsHubs = 0, gsChunks = 0;
    // colored order: per colour set, its degree classes and its chunk range
    struct GsSetLayout {
        uint32_t lo[8], hi[8], g[8];
        int nBins;
        uint32_t chunk0, chunk1;
    };
    std::vector<GsSetLayout> gsSetLayout;

    // Gauss-Seidel order (prepareGS)
    bool gsReady = false, gsColored = false;
    uint32_t gsPairK = 0;
    size_t gsDeferred = 0;
    gb::DevBuf<uint32_t> gsNat;          // natural order: list A | list B
    uint32_t gsNatA = 0, gsNatB = 0;
    std::vector<uint32_t> gsSetStart;    // colored: set k = ids [start[k], start[k+1])
    gb::DevBuf<uint32_t> rowGS, colGS, outdegGS;
    std::vector<uint32_t> gsNewId;
    gb::DevBuf<uint32_t> gsNewIdDev;
    bool gsLastRun = false;
    int lastVariant = -1;
    int lastCur = 0;                     // rank buffer of the last run
    gb::StagedCopy staged;

    // blocked pull: packed (row in block << 16 | column in part) per edge,
    // grouped by row block then part; blkOff[k * nParts + p] starts tile
    // (k, p), in 16-byte words
    gb::DevBuf<uint32_t> blkEdges, blkOff, blkHubs;
    uint32_t nRowBlocks = 0, rowsPer = 0, nParts = 0, nBlkHubs = 0;
    bool blkReady = false;

    // cached CUDA graphs of iteration batches, by what their kernels' arguments
    // depend on (the damping factor's bits last); at most kPrGraphs of them
    std::map<std::tuple<int, int, int, int, int, int, int, uint32_t>, cudaGraphExec_t> graphs;
    int grid = 0;

    ~gb_pr();
    void invalidateGraphs();
    void prepareAdaptive(uint32_t smallMax, uint32_t largeMin);
    void prepareGS(uint32_t pairMaxOutdeg);
    void prepareSplit(bool vector);
    void prepareBlocked();
    gb_pr_result run(int variant, const gb_pr_options& o);
    void ranks(float* out);
    void ranks64(double* out);
};
