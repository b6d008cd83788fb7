// fd_kernels.cuh -- launch interface of the timestep kernels (fd_kernels.cu).
#pragma once
#include "fd_internal.cuh"

// resident blocks per SM the narrow-phase kernels' registers are cut for.  The
// selection and the predicate pass: latency-bound gathers, so as many resident
// warps as fit without spilling; the contact law: its loads are kept together,
// which takes 128 registers.
#ifndef FD_SELECT_MIN_BLOCKS
#define FD_SELECT_MIN_BLOCKS 4
#endif
#ifndef FD_CONTACT_MIN_BLOCKS
#define FD_CONTACT_MIN_BLOCKS 2
#endif
#ifndef FD_PROBE_MIN_BLOCKS
#define FD_PROBE_MIN_BLOCKS 4
#endif
#ifndef FD_SUM_MIN_BLOCKS
#define FD_SUM_MIN_BLOCKS 4
#endif

namespace fd {

// default launch shape of the narrow phase, blocks per SM: selection, predicate
// pass, contact law, pair sums.  One resident wave, but two for the law: the
// first wave's early blocks make room for the rest (262,144 bodies: 44.9 us,
// 48.3 with one wave, 46.1 with four; 65,003: 16.6, 16.6, 18.8).
constexpr int DEFAULT_SHAPE[4] = {FD_SELECT_MIN_BLOCKS, FD_PROBE_MIN_BLOCKS, 4, FD_SUM_MIN_BLOCKS};

// Everything one simulation keeps on the device.  Plain pointers; ownership
// and sizes live in the host-side Sim object (fd_api.cu).
struct PairListDev {
    // pairs of the current step (A-major segments, partners ascending)
    int* pairA;
    int* pairB;
    int* seg_off;      // per particle A: first pair
    int* seg_cnt;      // per particle A: number of pairs
    int* c_off;        // per pair: first contact
    int* c_cnt;        // per pair: number of contacts
    double* pf;        // per pair, RESULT: F, torque on A, torque on B
    int* n_pairs;      // device counter
    int cap_pairs;
    // previous step (history source)
    int* o_pairA;
    int* o_counters;   // previous step's counters: pairs, slots, contacts
    int* o_pairB;
    int* o_seg_off;
    int* o_seg_cnt;
    int* o_c_off;
    int* o_c_cnt;
    // contact slots of the current step: the nodes that passed the
    // single-precision filter, contiguous per pair; c_node is the global
    // boundary-node id of a contact and -1 for a slot that is none
    int* c_node;
    int* c_at;         // per slot that holds a contact: its place in c_hist and c_rec
    int* c_pair;       // pair of each slot
    int* c_hit;        // slots holding a contact, listed by the predicate pass
                       // for the contact-law pass (n_hits of them)
    int* c_k;          // node key of each slot: cluster-order index relative to
                       // the geometry (ascending within a pair)
    // The contacts lie side by side, not slot by slot: one slot in eight holds
    // one.  Per contact 20 doubles (five sectors): [0 .. 8] F, torque on A,
    // torque on B (of the mode's type), [10 .. 18] with records: contact point,
    // normal, overlap, normal and tangential energy
    double* c_rec;
    double4* c_hist;   // per contact: tangential spring, partner (int in w's low half)
    int4* p_aux;       // per pair: cell of B (x, y, z), first history slot
    int* p_hist_cnt;   // per pair: history slots
    int* r_next;       // per pair: the next pair (code) of its partner's list
    int* p_hit;        // per pair: 1 when a slot of it holds a contact
    int* n_slots;      // device counter: slots used
    int* n_hits;       // device counter: contacts (n_slots + 1)
    int cap_contacts;  // slot capacity
    int* c_test;       // pair cache, carried steps: the slots the bound does not
                       // skip, listed for the predicate pass (n_test of them)
    int* n_test;
    float* p_bound;    // pair cache, carried steps: per pair, how far the SDF can
                       // have moved at a node since the rebuild (pair_bound)
    float* c_phi0;     // pair cache: per slot, the node's signed distance to the
                       // partner at the last rebuild (rounded down; -inf when
                       // the predicate stopped before the distance)
    // previous contacts
    int* o_c_node;
    int* o_c_k;
    int* o_c_at;
    double4* o_c_hist;
};

// A pair's or bond's force and two torques: three vectors of four (the last
// unused), so that a body reads its two in one load each.  As nine numbers
// they were six loads of eight bytes, each at 32 places a warp.
constexpr int RESULT = 12;

constexpr int CONTACT_REC = 20, CONTACT_POINT = 10, CONTACT_NORMAL = 13, CONTACT_OVERLAP = 16, CONTACT_EN = 17,
              CONTACT_ES = 18;

// Reverse index over the particle-particle and ghost lists together: for each
// particle, the pairs in which it is the partner, as codes pair * 8 + kind,
// sorted by (owner, kind).
struct RevDev {
    int* cnt;
    int* off;
    int* code;
    int cap;
    // the build: per particle the head of a list of its pairs (build number
    // << 32 | code, next in PairListDev::r_next), and the codes placed so far
    unsigned long long* head;
    int* total;
    const unsigned int* build;  // the step's build number (the particle cell table's)
    // the index is built when gate is null, or when *gate or *gate2 (may be
    // null) is not 0: a step whose lists keep their pairs keeps their index
    const int* gate;
    const int* gate2;
};

struct ObjDev {
    int n;
    double3* pos;
    double3* vel;
    double3* angvel;
    double3* force;
    double3* torque;
    fd_quat* q;
    int* mat;
    int* geo;
    long long* hash;   // cell hash of the current step (-1 when not hashed)
    int* node_base;    // first global boundary node of each object
    float4* rot;       // 3 per object: rows of the rotation matrix, single
                       // precision, refreshed at every hashing (culling only)
};

struct GeoSetDev {
    int n;
    const FdGeo* geo;
    const FdGeo32* geo32;
    const double* sdf;
    const float* sdf32;
    // per grid point the four corner values (x, x + 1) of rows y and y + 1:
    // what an interpolation reads of one z plane, in one load (null: not kept)
    const double4* sdf_quad;
    const float4* sdf32_quad;
    const float* dist;
    const float* cellmin;
    const double3* nodes;     // cluster order
    const int* node_lid;      // original local index of each node (cluster order)
    const FdCluster* clusters;
    const float4* nodes32;      // cluster order, single precision (culling only)
    const float4* clus_sphere;  // per cluster: centre, radius (single precision)
    const int2* clus_range;     // per cluster: first node, node count
    double rmax;              // largest bounding radius over the set
    double grid_rmax;         // largest grid radius over the set
};

struct MatDev {
    const double* kn;
    const double* ks;
    const double* mu;
    const double* e;
};

// Cell table of one object set (hashGrid of buildHashStartEnd.cu:69-137): a
// list of the objects in each cell.  A grid of few cells keeps a head per
// cell; a grid of many cells (dense would be large next to the object count)
// keeps an open-addressing hash table of its occupied cells instead.  A head
// holds (build number << 32 | first object): a head of another build is
// empty.  There is one build number per list generation; each is newer than
// every number a head can hold when its step begins (fd_build.h keeps them from
// coming round).
struct CellTableDev {
    FdGrid g;
    int hashed;                 // 0: a head per cell, 1: hash table of occupied cells
    unsigned long long* head;   // per cell, or per table slot
    int* next;                  // per object: the next one in its cell, -1 for the last
    unsigned int* build;        // [2] build numbers
    int par;                    // the list generation of this step: build[par] is its number
    unsigned long long* hkey;   // hashed: cell key per table slot (~0: empty)
    unsigned long long hmask;   // hashed: table size - 1 (a power of two)
};

struct GhostDev {
    double3* pos;
    long long* hash;
    CellTableDev cells;
    int* occ;  // box of the cells holding ghost images: min x, y, z, max x, y, z
    // sector images only (null for the translated X/Y images, which share the
    // particle's orientation and velocity): orientation, velocity and the
    // single-precision rotation rows of each image
    fd_quat* q;
    double3* vel;
    float4* rot;
    // translated images under the pair cache: 1 where the particle has an
    // image this step (the images of a rebuild also cover the particles
    // within the skin of the image band, whose pairs the cache keeps)
    unsigned char* live;
};

struct BondDev {
    int n;
    const int* master;
    const int* slave;
    int* active;
    double3* point;
    const double* B;      // 4 per bond
    const double* radius;
    const double* L0;
    const double* ts;
    const double* coh;
    const double* mu;
    const double3* frames; // 8 per bond: mn1 mn2 mn3 mp sn1 sn2 sn3 sp
    double* energy;        // 6 per bond: Un Us Ub Ut sn ss
    double* out;           // per bond, RESULT: F, Ti, Tj
    const int* plist_off;  // per particle (n+1): bonds touching it
    const int* plist;      // bond id * 2 + side
    int* rec_active;       // adjoint recording (null when off): bond active at the step
    double* rec_rij;       // 3 per bond: bond vector rb_i - rb_j at the step
    double* rec_dn;        // 3 per bond: frame difference n1j - n1i at the step
};

// Adjoint recording of one list at one step, one entry per contact slot
// (null pointers when not recording).  The partner index Bp is the particle
// that takes the reaction (the image's particle for ghosts, -1 for walls).
struct AdjRec {
    int* hit;        // 1 when the slot holds a contact
    int* A;
    int* Bp;
    int* B;          // partner as listed (wall index for walls)
    int* geoB;       // partner geometry (in the wall set for walls)
    int* matB;       // partner material (a wall material for walls)
    int* nid;        // global boundary-node id of the contact
    int* hist;       // slot of the same contact in the previous step, -1 when none
    double* rel;     // 3 per slot: contact node minus partner centre, world frame
    double* vc;      // 3 per slot: relative velocity of A against the partner
    double* sprev;   // 3 per slot: sliding spring before this step's update
    double* qB;      // 4 per slot: partner orientation
    double* arm;     // 3 per slot: contact node minus A's centre, world frame
    int* wrap;       // per slot: periodic shifts of the force-side centres,
                     // (sAx + 1) + 3 (sAy + 1) + 9 (sBx + 1) + 27 (sBy + 1)
    int cap;         // slots the record holds
};

// Verlet neighbour list of the particle-particle broad phase: per particle A,
// up to NL_MAX partners B > A whose centre lay within rA + rB + skin at the
// last build, ascending, by minimum-image distance in periodic directions
// (so a particle that wraps keeps the partners it meets on the other side).
// Rebuilt when a particle moved more than skin / 2 since then (minimum image)
// or changed visibility (inside or outside the domain).  The per-step filter
// applies the raw-position tests of the cell search.
constexpr int NL_MAX = 64;
struct NlDev {
    double3* ref;   // positions at the last build
    int* vis;       // visibility (cell hash >= 0) at the last build
    int* cnt;       // partners per particle
    int* list;      // NL_MAX per particle
    int* ctrl;      // [0]: rebuild requested
    double skin;
    int periodic_x, periodic_y;  // distances and displacements by minimum image
};

// Pair cache of the particle-particle list.  The candidate pairs and the
// nodes that may pass the node predicate (the contact slots) are built with
// every culling margin widened by a positional skin, and kept while no
// particle has drifted by more than skin / 2 since that build: the drift of
// particle i is |c_i - c_i0| + 2 r_max * 2 sin(theta_i / 2), theta_i its
// rotation since the build, which bounds how far any node of a pair can move
// in its partner's body frame (pairs stay listed, nodes stay slotted, while
// the two drifts sum to less than the skin).  Every step still runs the
// exact double-precision predicate on every slot, so the contacts are the
// ones a full detection gives.  ctrl[0]: rebuild this step (set by the check
// or by the host), ctrl[1]: rebuilds so far, ctrl[2]: the last build
// overflowed its lists (the next step builds again).
struct PairCacheDev {
    double3* ref_pos;   // positions at the last build
    fd_quat* ref_q;     // orientations at the last build
    int* ref_vis;       // visibility (hashed) at the last build
    // ctrl: [0] rebuild this step, [1] rebuilds so far, [2] the last build
    // overflowed the particle-particle lists, [3] rebuild at the next step,
    // [4] the translated ghost lists of this step are built, and without the
    // cache's skin (a particle wrapped, or an image outside the domain's
    // other directions), [7] rebuild requests of this step, moved to [3] at
    // its end
    int* ctrl;
    float* drift;       // per particle: the drift bound since the last build (rounded up)
    float4* disp;       // per particle: displacement since the last build (x, y, z) and
                        // the rotation part of the drift bound (rounded up)
    double skin;
    double reach;       // largest lever arm of a rotation in the drift bound:
                        // 2 r_max, or a larger SDF-grid radius
    // walls (the particle-wall list): state and cell at the last build, and
    // their drift bounds and displacements as for the particles (rotation
    // lever arm: the wall's SDF-grid radius)
    double3* wref_pos;
    fd_quat* wref_q;
    long long* wref_hash;
    float* wdrift;
    float4* wdisp;
};

struct StepArgs {
    AdjRec rec;      // recording of the list being launched (rec.hit null: off)
    double dt;
    double probe;      // contact when overlap >= -probe (0 in a timestep)
    int periodic_x, periodic_y;
    int sector;      // sector periodicity (the force side of particle and wall contacts folds bodies)
    int records;
    double skin;       // positional skin of the culling stages (the pair cache; 0 without it)
    const int* gate;   // pair cache: the list is built only when *gate or *gate2 (may be
    const int* gate2;  // null) is not 0, and carried otherwise (gate null: always built)
    const float* drift;  // pair cache: per-particle drift bounds (see PairCacheDev)
    const float4* disp;  // pair cache: per-particle displacements (see PairCacheDev)
    const float* driftB; // the partners' drift bounds and displacements when they
    const float4* dispB; // are walls (null: the particles')
    const int* noskin;   // non-null and nonzero: this step's selection takes no skin
    // launch shape of the narrow phase, in blocks per SM (0: the default):
    // selection, predicate pass, contact-law pass, pair sums
    int shape[4];
    unsigned int* flags;
    unsigned long long* stats;  // optional: pairs, clusters, clusters kept, contacts (narrow kernels)
};

// contiguous copy of a list's contacts, in (node, partner) order
struct ContactViewDev {
    double* point;     // 3 per contact
    double* normal;    // 3 per contact
    double* overlap;
    double* en;
    double* es;
    double* spring;    // 3 per contact
    int* master;       // global boundary node
    int* slave;        // partner
};
// a list's contacts packed for the host: ids (node, partner) and the wanted
// fields (null: not wanted)
struct ContactPackDev {
    int2* id;
    double *point, *normal, *overlap, *spring, *en, *es;
};
// the bonds' interleaved per-bond parameters and state as one array per field
struct BondViewDev {
    double* B[4];       // B1 .. B4
    double* energy[6];  // Un, Us, Ub, Ut, maximum normal stress, maximum shear stress
    double3* frames[8]; // master n1 n2 n3 point, slave n1 n2 n3 point (body frames)
};

// the tables of cell faces of one grid at off in the pools (quad may be null)
void launch_sdf_quads(const double* sdf, const float* sdf32, double4* quad, float4* quad32, long long off, int3 size,
                      cudaStream_t s);
// cell hash of each object (-1 outside the grid) and its single-precision
// rotation rows; build (non-null): the cell table's build numbers, renewed for
// a step of list generation par
void launch_hash(const ObjDev& O, const FdGrid& g, cudaStream_t s, unsigned int* build = nullptr, int par = 0);
// stable sort of n 64-bit keys (key 0 .. num_keys - 1, or negative: last) on
// the stream: out_idx gets the permutation, out_key the sorted keys (~0 for
// the negative ones).  Scratch: key_b (n), idx_b (n), bcount and bscan_tmp
// sized by radix_sort_scratch.
void radix_sort_keys(const long long* keys, int n, long long num_keys, unsigned long long* out_key, int* out_idx,
                     unsigned long long* key_b, int* idx_b, int* bcount, int* bscan_tmp, cudaStream_t s);
// ints needed for bcount and bscan_tmp for n keys
void radix_sort_scratch(int n, size_t& bcount_ints, size_t& bscan_ints);
// The periodic wraps (positions into dst, which may be P.pos) and the
// translated images gh[d] with on[d] (X, Y, XY).  Under the pair cache (ctrl
// non-null) a wrap requests the uncached ghost stage this step and a rebuild
// at the next; particles within ext_skin of the image band get images too
// (GhostDev::live marks the true ones); an image outside the domain in a
// direction it is not translated along (the reference hashes it into a clamped
// cell) makes this step's ghost stage uncached.
void launch_images(const ObjDev& P, double3* dst, const GhostDev* gh, const int* on, double ext_skin, int* ctrl,
                   cudaStream_t s);
// empty occupied-cell box of an image table (before the images are built)
void reset_image_box(int* occ, cudaStream_t s);
// sector periodicity: turn bodies that left the quarter sector back in, then
// build the three turned image sets (R90, R180, R270)
void launch_sector_wrap(ObjDev& P, const FdGrid& g, cudaStream_t s);
void launch_sector_images(const ObjDev& P, GhostDev* R, cudaStream_t s);

// What the lists of a step share, and one list of it
struct StepShared {
    int n;                   // particles
    GeoSetDev G, GW;
    MatDev M, MW;
    ObjDev W;
    FdGrid pgrid, wgrid;
    CellTableDev T;          // the particles' cell table
    // null: every wall; else per particle the first wall and the wall count it
    // may meet (a batch of simulations tiled into one)
    const int2* wall_range;
    RevDev R;
    int with_force;
    bool mixed;              // single-precision contact law, bond law and force sums
};
struct ListArgs {
    int kind;
    ObjDev P;                // the particles (image lists: at their wrapped positions)
    GhostDev gh;
    PairListDev L;
    StepArgs a;
};
// The stages of n lists, each stage one launch for all of them.  broad: cell
// tables and candidate pairs (nl non-null: the particle-particle list's come
// from the neighbour list; both give the same pairs).  narrow: contact slots,
// predicate, contact law, pair sums.  Under the pair cache (a.gate) a list
// that is not built this step keeps the pairs and slots of its last build.
void launch_broad(const ListArgs* lists, int n, const StepShared& c, NlDev* nl, cudaStream_t s);
void launch_narrow(const ListArgs* lists, int n, const StepShared& c, cudaStream_t s);
// end of a step's detection: the reverse index, and the pair cache's (pc
// non-null) layouts, references (refs: not yet taken by launch_cache_refs) and
// flags; done: a zeroed counter; flags: the error flags
void launch_step_end(const ObjDev& P, const ObjDev& W, const PairListDev* lists, const int* active, const RevDev& R,
                     const PairCacheDev* pc, bool cached_ghosts, bool refs, unsigned int* done, unsigned int* flags,
                     cudaStream_t s);
// the references of the pair cache, on a step that builds its lists
void launch_cache_refs(const ObjDev& P, const ObjDev& W, const PairCacheDev& pc, cudaStream_t s);
// parts of launch_advance and launch_small_advance: a step's force sums over
// its lists and bonds; its second half kick; the next step's first half kick,
// drift (walls too), hashes and, with pc, pair-cache checks, for a step of list
// generation par.  wrapped (may be null): the positions after the periodic
// wraps, which replace P.pos.  occ: the image tables' boxes to reset.
enum { STEP_SUM = 1, STEP_BACK = 2, STEP_FRONT = 4 };
void launch_advance(const StepShared& c, const ObjDev& P, const PairListDev* lists, const int* active, const BondDev& B,
                    const double3* wrapped, double3 gravity, double dt, const PairCacheDev* pc, int* const* occ,
                    int par, int parts, cudaStream_t s);
// Small sets (dense cell table, no neighbour list, pair cache or images): a
// step's detection, contact forces and pair sums of the particle-particle and
// particle-wall lists in one launch.  The cell table and both lists' counters
// (zero) are those launch_small_advance left; r_head (-1 per particle)
// collects each partner's pairs for its sum, own (6 per particle) the sums of
// each particle's own pairs.  a.rec: the record of the
// particle-particle list, recw of the particle-wall list.
void launch_small_pairs(const ObjDev& P, const GeoSetDev& G, const MatDev& M, const ObjDev& W, const GeoSetDev& GW,
                        const MatDev& MW, const FdGrid& pgrid, const FdGrid& wgrid, const CellTableDev& T,
                        const PairListDev& Lp, const PairListDev& Lw, const StepArgs& a, const AdjRec& recw,
                        const int2* wall_range, int* r_head, void* own, bool mixed, cudaStream_t s);
// launch_advance for a small set; its front also fills the cell lists T and
// zeroes the next lists' counters
void launch_small_advance(const ObjDev& P, const GeoSetDev& G, const ObjDev& W, const FdGrid& pgrid,
                          const FdGrid& wgrid, const PairListDev& Lp, const BondDev& B, const CellTableDev& T,
                          int* r_head, const void* own, int* zero_p, int* zero_w, double3 gravity, double dt,
                          bool mixed, int parts, cudaStream_t s);
// mixed: single-precision contact law, bond law and force sums
void launch_bonds(const ObjDev& P, BondDev& B, bool mixed, cudaStream_t s);
// the n contacts of a list (keys and sort scratch of the list's slot
// capacity; max_key bounds node << 32 | partner) into the view
void launch_contact_view(const PairListDev& L, long long* keys, int* order, unsigned long long* skey,
                         unsigned long long* key_b, int* idx_b, int* bcount, int* bscan, long long n,
                         long long max_key, const ContactViewDev& v, cudaStream_t s);
void launch_bond_view(const BondDev& B, const BondViewDev& v, cudaStream_t s);
// the contacts of a list, at most count, in no order; at: how many there are
void launch_pack_contacts(const PairListDev& L, const ContactPackDev& v, int* at, int count, cudaStream_t s);

// Kernel launches of the calling thread are counted into *c (null: not
// counted); the library points it at the calling simulation's counter for
// the duration of each call.  count_launch() counts one launch made
// elsewhere (the adjoint kernels).
void set_launch_counter(long long* c);
// whether the calling thread launches a step's kernels ahead of one another's
// end (default) or not (while it records a graph); see launch_ahead
void set_launch_ahead(bool on);
void count_launch();

// exclusive scan of n ints (out may alias in); returns needed tmp ints when tmp == nullptr
size_t scan_tmp_size(long long n);
void scan_exclusive(const int* in, int* out, long long n, int* tmp, cudaStream_t s);
// inclusive scan of n ints; tmp as for scan_exclusive
void scan_inclusive(const int* in, int* out, long long n, int* tmp, cudaStream_t s);

}  // namespace fd
