// engine.cuh -- host-side engine of one device-resident particle system.
#pragma once

#include <string>
#include <vector>

#include "device.cuh"
#include "error.cuh"
#include "k_ppe.cuh"

namespace mps {

// Growable device array; contents are not preserved on growth.
template <class T>
struct DevArray {
    T *p = nullptr;
    size_t n = 0;
    DevArray() = default;
    DevArray(const DevArray &) = delete;
    DevArray &operator=(const DevArray &) = delete;
    ~DevArray() { drop(); }
    static size_t room(size_t m) { return m + m / 8 + 16; }
    void reserve(size_t m)
    {
        if (m <= n) return;
        drop();
        size_t want = room(m);
        MPS_CUDA(cudaMalloc((void **)&p, want * sizeof(T)));
        n = want;
    }
    // storage that a DevGroup owns
    void place(void *q, size_t m)
    {
        drop();
        p = (T *)q;
        n = m;
        owned_ = false;
    }
    operator T *() const { return p; }

private:
    bool owned_ = true;
    void drop()
    {
        if (p && owned_) cudaFree(p);
        p = nullptr;
        n = 0;
        owned_ = true;
    }
};

// Arrays that are sized together and share one allocation (an allocation costs
// 0.3 ms and up to 30 ms in a busy process, whatever its size, and a session
// holds about a hundred arrays).  `list` calls its argument with every array
// of the group and the elements it needs; contents are not preserved on growth.
class DevGroup {
public:
    DevGroup() = default;
    DevGroup(const DevGroup &) = delete;
    DevGroup &operator=(const DevGroup &) = delete;
    ~DevGroup() { if (mem_) cudaFree(mem_); }
    template <class List>
    void reserve(List list)
    {
        bool grow = false;
        size_t bytes = 0;
        list([&](auto &a, size_t m) {
            grow = grow || m > a.n;
            bytes += size(a, m);
        });
        if (!grow) return;
        list([&](auto &a, size_t) { a.place(nullptr, 0); });
        if (mem_) cudaFree(mem_);
        mem_ = nullptr;
        MPS_CUDA(cudaMalloc((void **)&mem_, bytes));
        char *q = mem_;
        list([&](auto &a, size_t m) {
            a.place(q, a.room(m));
            q += size(a, m);
        });
    }

private:
    char *mem_ = nullptr;
    template <class T>
    static size_t size(const DevArray<T> &a, size_t m)
    {
        return (a.room(m) * sizeof(T) + 255) & ~(size_t)255;
    }
};

class EngineBase {
public:
    virtual ~EngineBase() = default;
    virtual int dim() const = 0;
    virtual void update_params(const mps_params_t &p) = 0;
    virtual void upload_aos(const void *aos, int num) = 0;
    virtual void download_aos(void *aos, int num) = 0;
    virtual void upload_soa(const double *pos, const double *vel, const int *type, int num) = 0;
    virtual void download_pressure(double *p, int num) = 0;
    virtual void compute_initial_params(double *n0, double *lambda, int *n0_count) = 0;
    virtual void set_initial_params(double n0, double lambda, int n0_count) = 0;
    virtual void neighbor_search() = 0;
    virtual void step(int nsteps) = 0;
    virtual void step_with_list(const int *nb, const int *cnt, int max_nb) = 0;
    virtual void get_neighbor_list(int *nb, int *cnt, int max_nb) = 0;
    virtual void get_cell_index(int *cell) = 0;
    virtual void get_cell_links(int *head, int *next, int total) = 0;
    virtual void set_precision(int precision) = 0;
    virtual void get_ppe(int *eq_idx, int *row_ptr, int *col, double *val, double *b, int *n_eq,
                         long long *nnz) = 0;
    virtual void run_stage(int stage, const int *nb, const int *cnt, int max_nb, double arg) = 0;
    // the last step's PPE and IC(0) preconditioner in the solver's numbering
    virtual void get_ic0(int *row_ptr, int *col, double *A, double *F, double *b, int *n_eq, long long *nnz) = 0;
    virtual void get_cell_blocks(int *cells, int *inv_off, double *inv, int *colour_rows, int *ncells,
                                 long long *ninv) = 0;
    virtual void apply_preconditioner(const double *r, double *z) = 0;
    virtual cudaStream_t stream() const = 0;
    // differentiation form: checkpoints and the adjoint of one step
    virtual size_t state_bytes() const = 0;
    virtual void state_save(void *dst) = 0;
    virtual void state_load(const void *src) = 0;
    virtual void adjoint_seed(const double *lam_pos, const double *lam_vel) = 0;
    virtual void adjoint_pressure_seed(const double *dLdP, int num) = 0;
    virtual void step_adjoint() = 0;
    virtual void adjoint_get(double *lam_pos, double *lam_vel, double *grad_gravity, double *grad_viscosity,
                             double *grad_drive) = 0;
    bool profiling = false;
    mps_metrics_t met{};
    std::string last_error;
};

EngineBase *make_engine(const mps_params_t &p, int capacity);

}  // namespace mps
