// Host-side driver of the D3 pipeline: model tables, lattice images, device
// workspace and the launch sequence of one evaluation.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "d3_device.cuh"

#ifndef DIRECT_MAX_ATOMS
#define DIRECT_MAX_ATOMS 256
#endif
#ifndef DIRECT_MAX_TOTAL
#define DIRECT_MAX_TOTAL 2048
#endif

namespace d3 {

struct Cutoffs {
    // realspace_cutoff defaults (cutoff.f90:26-38)
    double disp2 = 60.0, disp3 = 40.0, cn = 40.0, width2 = 0.0, width3 = 0.0;
};

struct Error : std::runtime_error {
    using std::runtime_error::runtime_error;
};

// Lattice translations within rthr (get_lattice_points, cutoff.f90:140-227).
// lattice[3][3] holds one vector per row; periodic[3].
// rep (or null): the translations run over -rep[k]..rep[k] along vector k.
std::vector<double> lattice_points(const double* lattice, const bool* periodic, double rthr, int* rep = nullptr);

// Wrap positions into the central cell (wrap_to_central_cell, utils.f90:29-64).
void wrap_to_central_cell(int nat, double* xyz, const double* lattice, const bool* periodic);

// True if two atoms are closer than 1e-9 Bohr (verify_structure, api.f90:1517-1530).
bool has_overlapping_atoms(int nat, const double* xyz);

// Species set and the per-species D3 model tables (new_d3_model, model.f90:87-181).
struct ModelTables {
    std::vector<int> num;            // atomic number per species
    std::vector<double> rcov, r4r2, refcn, c6ref, rvdw;
    std::vector<float> c6ref_f;
    std::vector<int> nref;
    int nid() const { return (int)num.size(); }
};

class Engine {
public:
    // nsys systems with natoms[s] atoms each; numbers concatenated.
    // lattices[nsys][9] and periodic[nsys][3] may be null (molecules).
    Engine(int nsys, const int* natoms, const int* numbers, const double* lattices,
           const bool* periodic, int device = -1);
    ~Engine();
    Engine(const Engine&) = delete;
    Engine& operator=(const Engine&) = delete;

    int nsys() const { return nsys_; }
    int natoms() const { return natoms_; }
    const ModelTables& tables() const { return tab_; }
    const std::vector<int>& atom_off() const { return atom_off_; }
    bool periodic_any(int sys) const;
    const double* lattice(int sys) const { return &lat_[9 * sys]; }
    const bool* periodic(int sys) const { return &per_[3 * sys]; }

    void set_cutoffs(const Cutoffs& c) { cut_ = c; images_valid_ = false; }
    const Cutoffs& cutoffs() const { return cut_; }
    void set_ghost(const std::vector<uint8_t>& ghost);
    void set_partition(int part, int nparts, bool cn_partitioned);
    void set_precision(int mixed) { mixed_ = mixed != 0; }
    bool mixed() const { return mixed_; }
    void set_counting(bool on) { counting_ = on; }
    void counts(long long out[3]) const;
    // Replace the lattices (host, [nsys][9]); images are rebuilt lazily.
    void set_lattices(const double* lattices);

    // Evaluate from host buffers (positions already wrapped).  Blocking.
    void evaluate_host(const Damp& d, const double* positions, double* energies, double* gradient,
                       double* sigma9);
    // Evaluate from device buffers on `stream` (the caller's stream, used as
    // given: 0 is the legacy default stream).  Asynchronous.
    void evaluate_device(const Damp& d, const double* d_positions, double* d_energies,
                         double* d_gradient, double* d_sigma9, double* d_param_grad,
                         cudaStream_t stream);
    // Pairwise decomposition from host buffers (positions already wrapped),
    // FP64 and without the work partition (get_pairwise_dispersion_v2):
    // energy2 and energy3 receive [n_s][n_s] per system, one system after the
    // other.  Blocking.
    void pairwise_host(const Damp& d, const double* positions, double* energy2, double* energy3);
    // Analytic Hessian [3n][3n] of a batch of one structure from host
    // positions (already wrapped), FP64 (get_dispersion_hessian); the work
    // partition splits the pair and triple loops.  Blocking.
    void hessian_host(const Damp& d, const double* positions, double* hessian);

    cudaStream_t stream() const { return stream_; }

    // Captured launch sequence.  With the graph on, an evaluation replays one
    // CUDA graph of the whole pipeline (sort, CN, weights, two-body, three-body
    // blocks and sum, chain rule, reductions) from engine-owned input/output
    // buffers.  The first evaluation of a (parameters, derivatives, tuning)
    // key runs the ordinary sequence, which sizes the three-body blocks, and
    // then captures the graph with 25% headroom on those buffers; a replay
    // whose blocks outgrow them is detected by a device flag and evaluated
    // again without the graph, and the graph is captured anew.
    void set_graph(bool on);
    bool graph() const { return graph_on_; }
    // kernel launches of one replay of the captured graph (0 before the first capture)
    long long graph_kernels() const { return graph_valid_ ? graph_kernels_ : 0; }

    // Partitioned evaluation over several processes (the reference's MPI
    // path, disp.f90:120-171 with a reducer, and mpi.f90): this engine
    // evaluates part `part` of `nparts` of every pair and triple loop,
    // including the CN and chain-rule loops, and calls `fn` to sum a device
    // buffer over all parts in place: the CN, then dE/dCN, then the results
    // [energies | parameter derivatives | virials | gradient] in one call.
    // `fn` is called on the host between launches and must order its work on
    // the given stream (a collective enqueued there, or a synchronisation
    // before a host exchange); it returns 0 on success.  All parts must have
    // the same systems, positions, parameters and launch shapes.  fn = null
    // ends the partition.  Not combinable with the captured graph.
    using Reducer = int (*)(double* buffer, int count, void* stream, void* user);
    void set_reducer(Reducer fn, void* user, int part, int nparts);

    // Launch shapes (spatial sort cell, items per tile pair, resident triple
    // blocks per SM).  autotune() times the candidates on the given device
    // positions and keeps the fastest; it returns that time in ms.
    void set_tuning(const Tuning& t);
    const Tuning& tuning() const { return tune_; }
    double autotune(const Damp& d, const double* d_positions, bool grad, cudaStream_t stream);
    // Device buffer of natoms x 3 positions owned by the engine (autotune input).
    double* input_buffer();

    // Per-stage device times of the last evaluation (ms), recorded with CUDA
    // events when profiling is on.  Stages: see kStageNames.
    static constexpr int kStages = 7;
    // stage_times() also returns, after the stages, the time of the two-body
    // tile-pair kernel alone and of the three-body triple kernels alone
    static constexpr int kTimes = kStages + 2;
    void set_profiling(bool on) { profiling_ = on; }
    void stage_times(double out[kTimes]);

private:
    void build_tables(const int* numbers);
    void ensure_images(cudaStream_t stream);
    void ensure_workspace(bool grad, bool param_grad, bool threebody);
    void upload_pair_table(const Damp& d, cudaStream_t stream);
    void make_views(Batch& b, Species& s) const;
    bool cn_single_chunk() const;
    static constexpr size_t kCnStoreCap = size_t(768) << 20;   // bytes of stored chain-rule sums at most
    static constexpr int kFusedWeightsMaxAtoms = 65536;          // CN gather fused with weights and species vectors
    unsigned char *d_cn_store_ = nullptr, *d_cn_store_ok_ = nullptr;
    size_t cn_store_cap_ = 0;
    void order_atoms(const Damp& d, const double* d_positions, const Batch& b, bool mixed, cudaStream_t stream);
    double* d_hs_ = nullptr;             // Hessian scratch and result
    double* d_rvdw_ = nullptr;           // [nid][nid] van der Waals radii (Hessian damping kernels)
    std::vector<int> img_off_host_;      // host copy of the image offsets
    double* d_pw_ = nullptr;             // pairwise decomposition: C6, energy2, energy3 (3 x sum n_s^2)
    long long* d_pw_off_ = nullptr;      // [2][nsys] first pair of each system, first pair and translation
    std::vector<long long> pw_off_;      // its host copy
    // pair factors of the triples: kept with the engine up to 256 MB, above that for the call
    static constexpr size_t kPwKeep = size_t(256) << 20;
    double* d_pw_mp_ = nullptr;
    size_t pw_mp_len_ = 0;
    void run(const Damp& d, const double* d_positions, double* d_energies, double* d_gradient,
             double* d_sigma9, double* d_param_grad, bool grad, cudaStream_t stream);
    template <class T> T* dev_alloc(size_t n);
    template <class T, class C> void regrow(T*& p, C& cap, size_t n);

    void reduce(double* buffer, int count, cudaStream_t stream);
    Reducer reducer_ = nullptr;
    void* reducer_user_ = nullptr;
    double* d_red_ = nullptr;    // [nsys | 5 nsys | 9 nsys | 3 natoms] results of this part

    // graph state
    struct GraphKey {
        Damp damp;
        Cutoffs cut;
        Partition part;
        Tuning tune;
        int grad, pg, counting, mixed, cn_part;
    };
    GraphKey make_key(const Damp& d, bool grad, bool pg) const;
    void run_graphed(const Damp& d, bool grad, bool pg, cudaStream_t stream);
    void capture(const Damp& d, const GraphKey& key, bool grad, bool pg);
    void drop_graph();
    // two-body tile-pair units
    PairUnits pu_;
    int2* d_units_ = nullptr;
    int* d_unit_base_ = nullptr;
    std::vector<int> sys_natoms_;
    int max_split_ = 4;                  // items per tile pair the slots are sized for
    int auto_split(int least) const;
    static constexpr int kDiagonalMaxAtoms = 256;
    bool diagonal_walks() const;
    int pair_split() const;              // items per tile pair of the two-body sweep
    int cn_split() const;                // items per tile pair of the CN sweeps
    bool any_periodic_ = false;          // a system has a periodic direction
    // systems small enough for the direct pair kernels (see direct_pairs)
    static constexpr int kDirectMaxAtoms = DIRECT_MAX_ATOMS;
    static constexpr int kDirectMaxTotal = DIRECT_MAX_TOTAL;
    bool small_systems() const;
    bool direct_pairs(const Damp& d, bool pg) const;
    bool graph_on_ = false, capturing_ = false, graph_valid_ = false;
    cudaGraphExec_t graph_exec_ = nullptr;
    long long graph_kernels_ = 0;
    GraphKey graph_key_{};
    unsigned long long alloc_epoch_ = 0, graph_epoch_ = 0;
    int* d_guard_ = nullptr;
    int* h_guard_ = nullptr;     // pinned
    double* d_pg_out_ = nullptr;
    Tuning tune_;
    int sms_ = 0;

    int device_ = 0;
    int nsys_ = 0, natoms_ = 0, max_sys_atoms_ = 0;
    std::vector<int> atom_off_, sys_of_atom_, local_, sp_;
    std::vector<int> zid_;               // species index inside the own system, from 1
    std::vector<double> lat_;
    std::vector<bool> per_storage_;
    std::unique_ptr<bool[]> per_;
    std::vector<uint8_t> ghost_;
    ModelTables tab_;
    Cutoffs cut_;
    Partition part_;
    bool cn_partitioned_ = false;
    bool mixed_ = false;
    bool counting_ = false;
    bool profiling_ = false;
    cudaEvent_t ev_[kStages + 1] = {};
    cudaEvent_t kev_[4] = {};            // two-body kernel, triple kernels: begin, end
    bool kev3_recorded_ = false;
    bool ev_recorded_ = false;
    bool images_valid_ = false;
    Damp last_damp_{};
    bool pair_valid_ = false;

    cudaStream_t stream_ = nullptr;
    std::vector<void*> allocations_;
    // static device data
    int *d_sys_of_atom_ = nullptr, *d_atom_off_ = nullptr, *d_local_ = nullptr, *d_sp_ = nullptr;
    uint8_t* d_ghost_ = nullptr;
    int* d_img_off_ = nullptr;
    double* d_img_ = nullptr;
    size_t img_capacity_ = 0;
    double *d_rcov_ = nullptr, *d_refcn_ = nullptr, *d_c6ref_ = nullptr, *d_pair_ = nullptr,
           *d_atm_r0_ = nullptr;
    float* d_c6ref_f_ = nullptr;
    int* d_nref_ = nullptr;
    // spatial order and tiles
    int ntiles_ = 0;
    int* d_tile_sys_ = nullptr;
    int* d_tile_off_ = nullptr;
    unsigned long long *d_keys_in_ = nullptr, *d_keys_out_ = nullptr;
    int *d_idx_in_ = nullptr, *d_perm_ = nullptr;
    int* d_identity_ = nullptr;           // 0 .. natoms - 1 (the order of the direct path)
    int *d_sp_sorted_ = nullptr, *d_local_sorted_ = nullptr, *d_zid_ = nullptr, *d_zid_sorted_ = nullptr;
    uint8_t* d_ghost_sorted_ = nullptr;
    double4* d_tiles_ = nullptr;
    int2* d_shape_ = nullptr;            // column order: slabs and columns per system
    void* d_sort_temp_ = nullptr;
    size_t sort_bytes_ = 0;
    // workspace
    double *d_x_ = nullptr, *d_y_ = nullptr, *d_z_ = nullptr;
    float4 *d_xhi_ = nullptr, *d_xlo_ = nullptr;
    Work work_{};
    bool ws_grad_ = false, ws_pg_ = false, ws_3b_ = false, ws_ready_ = false;
    double* d_pos_in_ = nullptr;
    double *d_energies_ = nullptr, *d_grad_out_ = nullptr, *d_sigma_ = nullptr;
    double *h_stage_ = nullptr;   // pinned staging: positions in, results out
    size_t h_stage_len_ = 0;
    // Pinned buffer for n result doubles (grown, kept with the engine) from the second
    // request on, or null: its allocation (6 ms for 0.4 and for 6 MB) takes longer than the
    // copies it saves in one call.  Null as well above kPinnedResults = 8 MB.  Below it stores to the buffer were the faster way at every
    // size (pairwise 700 atoms 5.3 -> 4.1 ms, Hessian of 330 2.69 -> 2.62 ms); above it
    // the kernels' work grows with the cube and pinned memory is not worth holding.
    static constexpr size_t kPinnedResults = size_t(1) << 20;
    double* pinned_results(size_t n);
    bool results_asked_ = false;
    double* h_results_ = nullptr;
    size_t h_results_len_ = 0;
    unsigned long long* d_counts_ = nullptr;
    // three-body
    // prepared: k_mol_pairs has ordered the tiles; launch_mol_finish takes the sums
    void run_three_body(const Batch& b, const Species& s, const Damp& d, const Config& c, Work& w,
                        cudaStream_t stream, bool prepared = false);
    int molecule_cluster(const Damp& d, bool pg) const;
    void run_molecules(const Batch& b, const Species& s, const Damp& d, const Config& c, int cluster,
                       const double* positions, double* energies, double* gradient, double* sigma9,
                       cudaStream_t stream);
    void* d_mol_fstore_ = nullptr;       // CN derivatives of small molecules' pairs
    void ensure_atm_layout(cudaStream_t stream);
    bool atm_compact(bool mixed) const;
    // FP32 triples up to this exponent: a pair's share (r0/r)^((alp + 2) / 3) of the damping
    // is bounded at 1e18 in FP32, which at 50 is passed below a twelfth of r0 (0.7 Bohr at
    // most), and at 100, where the bound would bite at a third of r0, costs the energy.
    static constexpr double kAtmMixedMaxAlp = 50.0;
    bool atm_mixed(const Damp& d) const { return mixed_ && d.alp <= kAtmMixedMaxAlp; }
    void free_block(void*& p);
    // blocks above this size are kept for the tile pairs in reach only
    static constexpr size_t kAtmDenseCap = size_t(1) << 30;
    // Systems of a batch whose blocks are held at a time: consecutive ones in processing
    // order with at most this many candidates (a larger system alone).  A candidate has 42
    // bytes of scratch, a kept block 1.5 or 3 KiB: 0.7 GB and, with a quarter in reach as
    // on periodic frames, 6 or 13 GB; the triples of a full group take a third of a second.
    static constexpr long long kAtmGroupCands = 1LL << 24;
    struct AtmGroup {
        int first, count;                // processing positions
        long long ncand, entries;        // candidate blocks, root list entries
        long long most;                  // largest number of tile images of a system
        bool operator==(const AtmGroup& o) const
        {
            return first == o.first && count == o.count && ncand == o.ncand && entries == o.entries && most == o.most;
        }
    };
    std::vector<AtmGroup> atm_groups_;
    void run_three_body_group(const AtmGroup& g, const Batch& b, const Species& s, const Damp& d, const Config& c,
                              const Work& w, cudaStream_t stream, bool prepared);
    std::vector<long long> c6mat_off_;   // dense [n_s][n_s] blocks of the pairwise decomposition
    long long c6mat_total_ = 0;
    int ntiles8_ = 0;
    std::vector<int> t8_off_;
    std::vector<int> img_rep_;           // [nsys][4] three-body translations of each system
    bool atm_layout_valid_ = false;
    AtmView atm_;
    long long *d_cand_off_ = nullptr, *d_cand_off_sys_ = nullptr, *d_list_off_ = nullptr;
    int* d_atm_group_ = nullptr;
    double4* d_pos8_ = nullptr;
    int* d_tile8_sys_ = nullptr;
    int4* d_atm_list_ = nullptr;
    int2* d_atm_range_ = nullptr;
    long long atm_list_cap_ = 0;
    int *d_atm_ord_ = nullptr, *d_atm_rep_ = nullptr, *d_t8_off_ = nullptr, *d_sub8_ = nullptr;
    double4* d_spheres8_ = nullptr;
    unsigned short* d_atm_mask_ = nullptr;
    long long atm_cand_cap_ = 0;
    int *d_atm_flag_ = nullptr, *d_atm_map_ = nullptr;
    unsigned char* d_scan_temp_ = nullptr;
    size_t scan_bytes_ = 0;
    long long atm_flag_cap_ = 0;
    unsigned char *d_atm_rec_ = nullptr, *d_atm_aux_ = nullptr;
    size_t atm_rec_cap_ = 0, atm_aux_cap_ = 0;        // bytes
    double* d_e3_ = nullptr;
    double* d_sig3_ = nullptr;
    unsigned long long *d_atm_queue_ = nullptr, *d_fxf_ = nullptr, *d_fxe_ = nullptr;
    int* h_atm_total_ = nullptr;         // pinned: kept blocks
    bool atm_ready_ = false;
    bool species_ready_ = false;   // PairUnits::U holds this evaluation's species vectors
};

}  // namespace d3
