// mpm_transfer.cuh — particle<->grid transfers, grid update and the implicit CG of one
// substep, as sm_103a kernels over the block-sparse grid of mpm_device.cuh.
//
// Work items ("chunks") are runs of at most `chunk` sorted particles inside one 4x4x4
// block. A chunk's stencils cover the 6x6x6 nodes from one below to one above its block,
// so every transfer kernel stages that tile in shared memory: P2G-type kernels accumulate
// into per-warp copies of it and flush them with one global vector atomic per touched
// node; G2P-type kernels load it once and gather from it. P2G writes each chunk's
// particles in cell order, and threads take them with a stride of chunk/32, so lanes of a
// warp sit in different cells and rarely scatter to the same nodes.
#pragma once
#include "mpm_device.cuh"

namespace mpm {

constexpr int TILE=6, TILE_N=TILE*TILE*TILE;
// Shared-memory layout of a 6x6x6 node tile: node (x, y, z) at x + TSY y + TSZ z, TILE_S
// words per channel. The z stride of 40 (not 36) spreads the cells of a block over the 32
// banks so that, with the cell order below, a warp's 32 scatter or gather addresses
// mostly fall in distinct banks.
constexpr int TSY=6, TSZ=40, TILE_S=5+5*TSY+5*TSZ+1;
__host__ __device__ constexpr int tile_addr(int tx,int ty,int tz){return tx+TSY*ty+TSZ*tz;}
__host__ __device__ constexpr int tile_addr(int t){return tile_addr(t%TILE,(t/TILE)%TILE,t/(TILE*TILE));}
constexpr int XFER_THREADS=128;   // CTA size of the transfer kernels = particles per work item
constexpr int NODE_THREADS=256;

// ---------- helpers ----------
__device__ __forceinline__ float tfma(float a,float b,float c){return fmaf(a,b,c);}
__device__ __forceinline__ double tfma(double a,double b,double c){return fma(a,b,c);}
__device__ __forceinline__ float tpow(float a,float b){return powf(a,b);}
__device__ __forceinline__ double tpow(double a,double b){return pow(a,b);}
__device__ __forceinline__ unsigned lane_bits_below(){unsigned m;asm("mov.u32 %0, %%lanemask_lt;":"=r"(m));return m;}
template<class T> __device__ __forceinline__ T sub_rn(T a,T b);
template<> __device__ __forceinline__ float sub_rn<float>(float a,float b){return __fsub_rn(a,b);}
template<> __device__ __forceinline__ double sub_rn<double>(double a,double b){return __dsub_rn(a,b);}
template<class T> __device__ __forceinline__ T add_rn(T a,T b);
template<> __device__ __forceinline__ float add_rn<float>(float a,float b){return __fadd_rn(a,b);}
template<> __device__ __forceinline__ double add_rn<double>(double a,double b){return __dadd_rn(a,b);}
template<class T> __device__ __forceinline__ T fmul_rn(T a,T b);
template<> __device__ __forceinline__ float fmul_rn<float>(float a,float b){return __fmul_rn(a,b);}
template<> __device__ __forceinline__ double fmul_rn<double>(double a,double b){return __dmul_rn(a,b);}

__device__ __forceinline__ void atomic_add_v3(V4<float>* p,float x,float y,float z,float w)
{atomicAdd(reinterpret_cast<float4*>(p),make_float4(x,y,z,w));}
__device__ __forceinline__ void atomic_add_v3(V4<double>* p,double x,double y,double z,double w)
{atomicAdd(&p->x,x);atomicAdd(&p->y,y);atomicAdd(&p->z,z);if(w!=0.) atomicAdd(&p->w,w);}

// Hides a value from the compiler's loop-invariant motion: the scatters' rounds loop mostly
// runs once, and the coefficients of all nine (x, y) columns hoisted out of it would take more
// registers than a thread has.
__device__ __forceinline__ void opaque(float& x){asm volatile("":"+f"(x));}
__device__ __forceinline__ void opaque(float2& x){asm volatile("":"+f"(x.x),"+f"(x.y));}
__device__ __forceinline__ void opaque(double& x){asm volatile("":"+d"(x));}

// Chunk geometry: particle range, block, scene and the 27 neighbour active indices.
template<class T> struct ChunkInfo {
    int s,e,scene;
    int b[3];        // block coordinates inside the scene
    long long gb;
};
// Block coordinates of global block gb of a scene (block ids have 26 bits: 32-bit divisions).
template<class T> __device__ __forceinline__ void block_coords(const SceneDev<T>& sc,long long gb,int* b)
{
    const unsigned lb=(unsigned)(gb-sc.block_base),n0=(unsigned)sc.nb[0],n1=(unsigned)sc.nb[1],q=lb/n0,q2=q/n1;
    b[0]=(int)(lb-q*n0);b[1]=(int)(q-q2*n1);b[2]=(int)q2;
}
// The geometry of work item c; lanes (threads) 0..26 of the caller fill nbr[27].
template<class T> __device__ __forceinline__ bool load_chunk(const DevState<T>& S,long long c,unsigned nc,unsigned nv,ChunkInfo<T>& ci,int* nbr,
                                                             int lane=-1)
{
    if(lane<0) lane=threadIdx.x;
    ci.s=S.chunk_start[c];
    ci.e=(c+1<nc)?S.chunk_start[c+1]:(int)nv;
    ci.gb=(long long)(S.keys[ci.s]>>6);
    ci.scene=scene_of_block(S.scene_block_base,S.n_scenes,ci.gb);
    const SceneDev<T>& sc=S.scenes[ci.scene];
    block_coords(sc,ci.gb,ci.b);
    if(lane<27){
        const int ox=lane%3-1,oy=(lane/3)%3-1,oz=lane/9-1;
        const long long g2=ci.gb+ox+(long long)sc.nb[0]*(oy+(long long)sc.nb[1]*oz);
        nbr[lane]=bit_set(S.bitmap,g2)?S.blockmap[g2]:-1;}
    return true;
}
// Tile node t (0..215) -> global node index, or -1 if its block is not active.
__device__ __forceinline__ long long tile_node(const int* nbr,int t)
{
    const int tx=t%TILE,ty=(t/TILE)%TILE,tz=t/(TILE*TILE);
    const int ox=(tx+3)/4-1,oy=(ty+3)/4-1,oz=(tz+3)/4-1;        // 0 -> -1, 1..4 -> 0, 5 -> +1
    const int idx=nbr[(ox+1)+3*(oy+1)+9*(oz+1)];
    if(idx<0) return -1;
    const int l=((tx+3)&3)|(((ty+3)&3)<<2)|(((tz+3)&3)<<4);
    return (long long)idx*64+l;
}
// Per-particle stencil data: tile coordinates of node c-1 and the weights along each axis.
template<class T> struct Stencil {
    int r[3];        // tile coordinate of the particle's cell (1..4)
    T w[3][3],dw[3][3];
};
// Stencil coordinates x = (X - (center(c) - dx))/dx in [0.5, 1.5) of a particle in local cell
// l of block b, evaluated in the same order as the reference.
template<class T> __device__ __forceinline__ void stencil_coord(const SceneDev<T>& sc,const int* b,unsigned l,const T* X,T* x)
{
    const int lc[3]={(int)(l&3u),(int)((l>>2)&3u),(int)(l>>4)};
#pragma unroll
    for(int a=0;a<3;++a){
        const int cell=4*b[a]+lc[a]-4;
        const T center=fmul_rn<T>(add_rn<T>((T)cell,(T)0.5),sc.dx[a]);
        const T xe=sub_rn<T>(X[a],sub_rn<T>(center,sc.dx[a]));
        x[a]=fmul_rn<T>(xe,sc.inv_dx[a]);}
}
template<class T> __device__ __forceinline__ void stencil_from_coord(const SceneDev<T>& sc,unsigned l,const T* x,Stencil<T>& st)
{
    st.r[0]=(int)(l&3u)+1;st.r[1]=(int)((l>>2)&3u)+1;st.r[2]=(int)(l>>4)+1;
#pragma unroll
    for(int a=0;a<3;++a) bspline_weights<T>(x[a],sc.inv_dx[a],st.w[a],st.dw[a]);
}
template<class T> __device__ __forceinline__ void make_stencil(const SceneDev<T>& sc,const int* b,unsigned key,const T* X,Stencil<T>& st)
{
    T x[3];stencil_coord(sc,b,key&63u,X,x);
    stencil_from_coord(sc,key&63u,x,st);
}
// Node centre of a grid node.
template<class T> __device__ __forceinline__ void node_center(const DevState<T>& S,const SceneDev<T>& sc,long long node,int blk,T* x)
{
    int b[3];block_coords(sc,S.active_gb[blk],b);
    const int l=(int)(node&63);
    const int c[3]={4*b[0]+(l&3)-4,4*b[1]+((l>>2)&3)-4,4*b[2]+(l>>4)-4};
#pragma unroll
    for(int a=0;a<3;++a) x[a]=((T)c[a]+(T)0.5)*sc.dx[a];
}
template<class T> __device__ __forceinline__ bool inside_barrier(const SceneDev<T>& sc,int b,const T* x)
{return (x[0]-sc.bs[b][0])*sc.bn[b][0]+(x[1]-sc.bs[b][1])*sc.bn[b][1]+(x[2]-sc.bs[b][2])*sc.bn[b][2]<T(0);}

// Particle order inside a work item for the scatter kernels: the item's n particles are
// split into 32 runs of `stride` = ceil(n/32) consecutive (cell-sorted) particles, lane L
// walks run L, and the CTA's warps take successive positions inside the runs. Lanes of a
// warp therefore sit about n/32 particles apart, i.e. in different cells for a full
// block, and their shared atomics rarely hit the same node.
#define FOR_INTERLEAVED(n,jvar) \
    for(int q_=(int)(threadIdx.x>>5),st_=((n)+31)>>5;q_<st_;q_+=(int)(blockDim.x>>5)) \
        for(int jvar=(int)(threadIdx.x&31)*st_+q_,ok_=1;ok_;ok_=0) if(jvar<(n))

// ---------- per-scene reductions inside node kernels ----------
struct SceneRed {
    unsigned long long mx[MAX_SCENES];
    unsigned long long cnt[MAX_SCENES];
};
__device__ __forceinline__ void red_init(SceneRed& R,int ns)
{for(int i=threadIdx.x;i<ns;i+=blockDim.x){R.mx[i]=0ull;R.cnt[i]=0ull;}}
template<class TR> __device__ __forceinline__ TR warp_sum(TR v){for(int o=16;o>0;o>>=1) v+=__shfl_xor_sync(0xffffffffu,v,o);return v;}
template<class TR> __device__ __forceinline__ TR warp_max(TR v){for(int o=16;o>0;o>>=1){TR u=__shfl_xor_sync(0xffffffffu,v,o);v=u>v?u:v;}return v;}
__device__ __forceinline__ unsigned long long dbits(double x){return (unsigned long long)__double_as_longlong(x);}
__device__ __forceinline__ double bitsd(unsigned long long b){return __longlong_as_double((long long)b);}
// Flush the CTA's per-scene partials (maximum, and the count when asked for) to the global
// accumulators, then let the last of the `parts` CTAs that take part (ticket) run `fin` for
// every scene; fin sees complete values. Returns true in every thread of that CTA.
template<bool USE_CNT,class F> __device__ __forceinline__ bool red_finish(SceneRed& R,int ns,SceneAcc* acc,unsigned* ticket,unsigned parts,F fin)
{
    __syncthreads();
    for(int i=threadIdx.x;i<ns;i+=blockDim.x){
        if(R.mx[i]) atomicMax(&acc[i].max0,R.mx[i]);
        if(USE_CNT&&R.cnt[i]) atomicAdd(&acc[i].count0,R.cnt[i]);}
    __threadfence();
    __shared__ bool last;
    __syncthreads();
    if(threadIdx.x==0) last=(atomicAdd(ticket,1u)==parts-1u);
    __syncthreads();
    if(!last) return false;
    __threadfence();
    for(int i=threadIdx.x;i<ns;i+=blockDim.x){
        volatile SceneAcc* a=acc+i;
        const unsigned long long m=a->max0,c=a->count0;
        a->max0=0ull;a->count0=0ull;
        fin(i,bitsd(m),c);}
    __syncthreads();
    if(threadIdx.x==0) *ticket=0u;
    return true;
}
// CTAs of the grid that get any of `work` items when each takes `per` at least; at least one
// (it runs the reduction's end). The others return at once: with a small scene's few dozen
// blocks, hundreds of CTAs would otherwise pass through the one ticket.
__device__ __forceinline__ unsigned taking_part(long long work,long long per)
{
    const long long n=(work+per-1)/per;
    return (unsigned)(n<1?1:n<(long long)gridDim.x?n:(long long)gridDim.x);
}

// A running sum per lane for the node kernels. FP32 terms go into an unevaluated pair by TwoSum
// (48 bits): an FP64 addition and its conversion take the FP64 pipe, at 1/64 of the FP32
// rate, longer than the node's memory traffic takes.
template<class T> struct NodeSum { T h=T(0);
    __device__ __forceinline__ void add(T x){h+=x;}
    __device__ __forceinline__ double value() const {return h;} };
template<> struct NodeSum<float> { float h=0.f,l=0.f;
    __device__ __forceinline__ void add(float x)
    {const float s=__fadd_rn(h,x),z=__fadd_rn(s,-h);l+=__fadd_rn(__fadd_rn(h,-__fadd_rn(s,-z)),__fadd_rn(x,-z));h=s;}
    __device__ __forceinline__ double value() const {return (double)h+(double)l;} };
// The sum of a warp's lanes. FP32 adds the lanes' pairs by the same TwoSum and converts once: an
// FP64 addition keeps the SM's FP64 units busy for 16 cycles a warp, and the five steps of
// four quantities took 1 us of a CG trip of a small scene.
__device__ __forceinline__ double warp_value(NodeSum<float> v)
{
#pragma unroll
    for(int o=16;o>0;o>>=1){
        const float h=__shfl_xor_sync(0xffffffffu,v.h,o),l=__shfl_xor_sync(0xffffffffu,v.l,o);
        v.add(h);v.l=__fadd_rn(v.l,l);}
    return v.value();
}
__device__ __forceinline__ double warp_value(NodeSum<double> v){return warp_sum<double>(v.h);}
// The reduction of kernels whose warps walk contiguous block ranges: a warp's last scene goes
// into its slot here, an earlier one (rare) straight to the accumulators; one warp joins the
// slots (mostly one scene) and adds them. Against per-scene shared arrays this spares a
// small scene the shared FP64 atomics and the loops over all scenes.
struct WarpParts { int scene[NODE_THREADS/32]; double sum[NODE_THREADS/32][3]; double mx[NODE_THREADS/32]; };
template<int NS> __device__ __forceinline__ void add_scene(SceneAcc* acc,int sc,const double* s,double mx)
{
#pragma unroll
    for(int k=0;k<NS;++k) if(s[k]!=0.) atomicAdd(&acc[sc].sum[k],s[k]);
    if(mx>0.) atomicMax(&acc[sc].max0,dbits(mx));
}
template<int NS,class T> __device__ __forceinline__ void flush_scene(WarpParts& W,SceneAcc* acc,int sc,bool last,const NodeSum<T>& a,const NodeSum<T>& b,
    const NodeSum<T>& c,T mx)
{
    const double s[3]={warp_value(a),NS>1?warp_value(b):0.,NS>2?warp_value(c):0.},m=(double)warp_max<T>(mx);
    if((threadIdx.x&31)!=0) return;
    if(!last){add_scene<NS>(acc,sc,s,m);return;}
    const int w=threadIdx.x>>5;
    W.scene[w]=sc;W.mx[w]=m;
#pragma unroll
    for(int k=0;k<NS;++k) W.sum[w][k]=s[k];
}
// As red_finish. Every warp has flushed its last scene (-1: none) into W.
template<int NS,class F> __device__ __forceinline__ bool parts_finish(const WarpParts& W,int ns,SceneAcc* acc,unsigned* ticket,unsigned parts,F fin)
{
    __shared__ bool last;
    __syncthreads();
    if(threadIdx.x<32){
        const int w=threadIdx.x,nw=blockDim.x>>5;
        const int sc=w<nw?W.scene[w]:-1;
        double s[3]={0.,0.,0.},m=0.;
        if(sc>=0){
#pragma unroll
            for(int k=0;k<NS;++k) s[k]=W.sum[w][k];
            m=W.mx[w];}
        const unsigned any=__ballot_sync(0xffffffffu,sc>=0);
        const int sc0=__shfl_sync(0xffffffffu,sc,any?__ffs(any)-1:0);
        if(__all_sync(0xffffffffu,sc<0||sc==sc0)){
            for(int o=NODE_THREADS/64;o>0;o>>=1){
#pragma unroll
                for(int k=0;k<NS;++k) s[k]+=__shfl_xor_sync(0xffffffffu,s[k],o);
                m=fmax(m,__shfl_xor_sync(0xffffffffu,m,o));}
            if(w==0&&any) add_scene<NS>(acc,sc0,s,m);}
        else if(sc>=0) add_scene<NS>(acc,sc,s,m);
        __threadfence();
        __syncwarp();
        if(w==0){last=(atomicAdd(ticket,1u)==parts-1u);if(last) *ticket=0u;}}
    __syncthreads();
    if(!last) return false;
    __threadfence();
    for(int i=threadIdx.x;i<ns;i+=blockDim.x){
        volatile SceneAcc* a=acc+i;
        double s[3]={0.,0.,0.};
#pragma unroll
        for(int k=0;k<NS;++k){s[k]=a->sum[k];a->sum[k]=0.;}
        const unsigned long long m=a->max0;
        a->max0=0ull;
        fin(i,s,bitsd(m));}
    return true;
}

// A warp's contiguous share [b, b1) of nb node blocks.
struct WarpRange {
    int b,b1;
    unsigned parts;          // CTAs with a block
    __device__ __forceinline__ explicit WarpRange(int nb)
    {
        const int nw=(int)(gridDim.x*(blockDim.x>>5)),gw=(int)(blockIdx.x*(blockDim.x>>5)+(threadIdx.x>>5));
        const int per=(nb+nw-1)/nw;
        b=gw*per<nb?gw*per:nb;b1=b+per<nb?b+per:nb;
        parts=taking_part(nb,(long long)max(per,1)*(blockDim.x>>5));
    }
};
// Exclusive prefix sum of one int per thread over the CTA (any blockDim up to 1024);
// *total receives the sum. Called by every thread.
__device__ __forceinline__ int cta_scan_int(int v,int* total)
{
    __shared__ int wsum[32];
    const int lane=threadIdx.x&31,w=threadIdx.x>>5,nw=(blockDim.x+31)>>5;
    int x=v;
#pragma unroll
    for(int o=1;o<32;o<<=1){const int y=__shfl_up_sync(0xffffffffu,x,o);if(lane>=o) x+=y;}
    if(lane==31) wsum[w]=x;
    __syncthreads();
    if(w==0){int t=lane<nw?wsum[lane]:0;
#pragma unroll
        for(int o=1;o<32;o<<=1){const int y=__shfl_up_sync(0xffffffffu,t,o);if(lane>=o) t+=y;}
        wsum[lane]=t;}
    __syncthreads();
    const int excl=x-v+(w>0?wsum[w-1]:0);
    *total=wsum[nw-1];
    __syncthreads();
    return excl;
}
// Last CTA of a convergence check (after its per-scene updates of S.cg): the list of the
// scenes that still iterate, for the next loop trip. One thread per scene (blockDim >=
// n_scenes); every thread of the CTA calls it.
template<class T> __device__ __forceinline__ void build_active_list(const DevState<T>& S)
{
    __syncthreads();
    const int i=threadIdx.x;
    int act=0,nc=0,nb=0;
    if(i<S.n_scenes&&!S.cg[i].done){const SceneRange r=S.srange[i];act=1;nc=r.c1-r.c0;nb=r.b1-r.b0;}
    if(S.n_scenes==1){                               // no scans for a single scene
        if(i==0){
            ActiveList* L=S.alist;
            L->scene[0]=0;L->cpre[0]=L->bpre[0]=0;L->n=act;
            if(act){L->cpre[1]=nc;L->bpre[1]=nb;}}
        return;}
    int na,ct,bt;
    const int pos=cta_scan_int(act,&na),cp=cta_scan_int(nc,&ct),bp=cta_scan_int(nb,&bt);
    ActiveList* L=S.alist;
    if(act){L->scene[pos]=i;L->cpre[pos]=cp;L->bpre[pos]=bp;}
    if(i==0){L->n=na;L->cpre[na]=ct;L->bpre[na]=bt;}
}
// The list staged in shared memory by every CTA of a loop-trip kernel.
struct ListSmem { int n; int scene[MAX_SCENES]; int pre[MAX_SCENES+1]; };
__device__ __forceinline__ void load_active_list(const ActiveList* L,ListSmem& sm,bool blocks)
{
    const int n=L->n;
    for(int k=threadIdx.x;k<=n;k+=blockDim.x){
        if(k<n) sm.scene[k]=L->scene[k];
        sm.pre[k]=blocks?L->bpre[k]:L->cpre[k];}
    if(threadIdx.x==0) sm.n=n;
    __syncthreads();
}
// Position j in the list with pre[j] <= w < pre[j+1] (w < pre[n]).
__device__ __forceinline__ int list_find(const ListSmem& sm,int w)
{
    int lo=0,hi=sm.n-1;
    while(lo<hi){const int mid=(lo+hi+1)>>1;if(sm.pre[mid]<=w) lo=mid;else hi=mid-1;}
    return lo;
}

// =====================================================================================
// K3: plasticity + P2G. Per particle: Precompute (MPM_Constitutive_Model.cpp:32-51,
// called at MPM_Example.cpp:563-571), then the scatter of m, m v (Rasterize,
// MPM_Example.cpp:520-537) and f = sum_p (m_p g w - V0 P Fe^T grad w) (Apply_Explicit_Force,
// MPM_Example.cpp:757-784). Reads the old particle buffer through the sort permutation and
// writes the new one, cell-ordered inside every work item, with its keys and the CG cache.
// =====================================================================================
// Shared-memory bytes of one FP64 P2G CTA: the warps' private tiles and (also k_items) the
// cell order of a work item of up to `chunk` particles (per-warp cell counts, slot -> item
// map, item cells).
template<class T> __host__ __device__ constexpr int p2g_tile_bytes(){return (XFER_THREADS/32)*7*TILE_S*(int)sizeof(T);}
__host__ __device__ constexpr int order_bytes(int chunk){return (XFER_THREADS/32)*64*4+64*4+((chunk*5+15)&~15);}
template<class T> __host__ __device__ constexpr int p2g_smem_bytes(int chunk){return p2g_tile_bytes<T>()+order_bytes(chunk);}

// Scatter order of a block's 64 cells: by the shared-memory bank of the cell's tile address
// (tile_addr mod 32), then by cell index. With TSZ = 40 every bank holds exactly two cells,
// so cells of even rank have 32 distinct banks, and so do cells of odd rank. A warp's lanes
// sit about two cells apart in this order (a full block has 8 particles per cell and the
// lanes are chunk/32 particles apart), so their tile addresses, and for every stencil
// offset the addresses of their nodes, fall in distinct banks.
struct CellRank { unsigned char rank[64],cell[64]; };     // rank of a cell, cell of a rank
constexpr CellRank make_cell_rank()
{
    CellRank r{};
    for(int l=0;l<64;++l){
        const int b=(l%4+TSY*((l/4)%4)+TSZ*(l/16))%32;
        int k=0;
        for(int m=0;m<64;++m){const int bm=(m%4+TSY*((m/4)%4)+TSZ*(m/16))%32;k+=(bm<b||(bm==b&&m<l))?1:0;}
        r.rank[l]=(unsigned char)k;r.cell[k]=(unsigned char)l;}
    return r;
}
static __device__ const CellRank cell_ranks=make_cell_rank();

// Storage order of a work item. Pass q of a warp gives lane L the cell-ordered slot
// k = L*stride + q (stride = ceil(np/32)), so the lanes of a warp sit about two cells
// apart. Slot (q, L) is stored at position run[q] + L, where run[q] counts the valid slots
// of the passes before q (the valid lanes of a pass are a prefix of the warp): a warp's
// loads and stores of one pass are contiguous. Called by warp 0; run has stride+1 entries
// (stride <= 128 for work items of up to 4096 particles).
__device__ __forceinline__ void chunk_runs(int np,int stride,int* run)
{
    const int lane=threadIdx.x&31;
    int c[4],tot=0;
#pragma unroll
    for(int u=0;u<4;++u){
        const int q=4*lane+u;const int r=np-q;
        c[u]=(q<stride&&r>0)?min(32,(r+stride-1)/stride):0;tot+=c[u];}
    int incl=tot;
#pragma unroll
    for(int o=1;o<32;o<<=1){const int v=__shfl_up_sync(0xffffffffu,incl,o);if(lane>=o) incl+=v;}
    int acc=incl-tot;
#pragma unroll
    for(int u=0;u<4;++u){const int q=4*lane+u;if(q<=stride) run[q]=acc;acc+=c[u];}
}

// Stable counting sort of a work item's particles by the scatter rank of their cell (the
// low 6 key bits through crank): on return inv[k] is the item position of the k-th
// particle in (rank, item position) order, cellv[j] the cell of item position j, and
// cnt[w][r] where warp w's particles of rank r begin. Warp w owns the item positions [w*seg,
// (w+1)*seg): it numbers its particles inside their cell (loc) and counts the ranks, a warp
// scan turns the counts into (rank, warp)-major offsets, and every particle is placed. The
// particles of a block keep their order from one substep to the next (the block sort is
// stable), so writing the new buffer in this order makes the chunk rank-sorted for the
// Hessian and G2P of this substep and nearly so for the next P2G. Returns the end of rank r
// in rank_end[r].
__device__ __forceinline__ void chunk_cell_order(const unsigned* keys,int s,int np,const unsigned char* crank,int (*cnt)[64],unsigned short* inv,
    unsigned short* loc,unsigned char* cellv,int* rank_end)
{
    const int lane=threadIdx.x&31,warp=threadIdx.x>>5,nw=blockDim.x>>5;
    for(int t=threadIdx.x;t<nw*64;t+=blockDim.x) (&cnt[0][0])[t]=0;
    __syncthreads();
    const int seg=(np+nw-1)/nw,b0=warp*seg,b1=min(np,b0+seg);
    const unsigned below=lane_bits_below();
    unsigned key=b0+lane<b1?keys[s+b0+lane]:0u;
    for(int g=b0;g<b1;g+=32){
        const int j=g+lane;const bool ok=j<b1;
        const unsigned cell=key&63u;
        key=j+32<b1?keys[s+j+32]:0u;
        const unsigned rk=crank[cell];
        // lanes of the same cell by six ballots (match.any costs more the more cells a warp has)
        unsigned peers=__ballot_sync(0xffffffffu,ok);
#pragma unroll
        for(int b=0;b<6;++b){const bool bit=(cell>>b)&1u;const unsigned m=__ballot_sync(0xffffffffu,bit);peers&=bit?m:~m;}
        const int before=ok?cnt[warp][rk]:0,rank=__popc(peers&below);
        __syncwarp();
        if(ok){
            cellv[j]=(unsigned char)cell;loc[j]=(unsigned short)(before+rank);
            if(rank==0) cnt[warp][rk]=before+__popc(peers);}
        __syncwarp();}
    __syncthreads();
    if(warp==0){
        const int c0=2*lane,c1=2*lane+1;
        int t0=0,t1=0;
        for(int w=0;w<nw;++w){t0+=cnt[w][c0];t1+=cnt[w][c1];}
        int incl=t0+t1;
#pragma unroll
        for(int o=1;o<32;o<<=1){const int u=__shfl_up_sync(0xffffffffu,incl,o);if(lane>=o) incl+=u;}
        int o0=incl-(t0+t1),o1=o0+t0;
        rank_end[c0]=o1;rank_end[c1]=incl;
        for(int w=0;w<nw;++w){
            const int a=cnt[w][c0],b=cnt[w][c1];
            cnt[w][c0]=o0;o0+=a;cnt[w][c1]=o1;o1+=b;}}
    __syncthreads();
    for(int j=b0+lane;j<b1;j+=32) inv[cnt[warp][crank[cellv[j]]]+loc[j]]=(unsigned short)j;
    __syncthreads();
}

// Pair table of a work item, for the kernels that handle two particles of one cell per lane.
// The particles of a cell are paired in slot order (an odd one stays alone); the pairs are
// listed level by level, the first pairs of all cells, then the second ones, and so on, the
// cells of a level with even scatter rank before those with odd rank. 32 consecutive
// pairs, one warp's pass, therefore lie in distinct cells whose tile addresses fall in
// distinct banks wherever a level has enough cells. Entry: positions of the two
// particles in the item (12 bits each), cell (6 bits), PAIR_TWO when there is a second one.
constexpr unsigned PAIR_TWO=1u<<30;
// Stored position of cell-ordered slot k of a work item (chunk_runs); rs = 1/stride. The
// quotient is exact: k + 1/2 lies at least 1/256 from a multiple of stride <= 128, in units of
// the quotient, and FP32 rounding of values below 4,096 stays under that.
__device__ __forceinline__ int slot_position(int k,int stride,float rs,const int* run)
{
    const int L=(int)(((float)k+0.5f)*rs);
    return run[k-L*stride]+L;
}
__device__ __forceinline__ unsigned pair_entry(int k,bool two,unsigned cell,int stride,float rs,const int* run)
{
    const int p0=slot_position(k,stride,rs,run),p1=two?slot_position(k+1,stride,rs,run):p0;
    return (unsigned)p0|((unsigned)p1<<12)|(cell<<24)|(two?PAIR_TWO:0u);
}
// Called by every warp of the CTA, which writes the levels warp, warp + nw, ...; rank_end[r] is
// the end of scatter rank r in the item's slot order and cell_of[r] its cell. Returns the
// number of pairs.
__device__ __forceinline__ int pair_table(const int* rank_end,const unsigned char* cell_of,int stride,const int* run,unsigned* out)
{
    const int lane=threadIdx.x&31,warp=threadIdx.x>>5,nw=blockDim.x>>5;
    const int e0=rank_end[2*lane],e1=rank_end[2*lane+1];
    int s0=__shfl_up_sync(0xffffffffu,e1,1);
    if(lane==0) s0=0;
    const unsigned below=lane_bits_below();
    const unsigned c0=cell_of[2*lane],c1=cell_of[2*lane+1];
    const float rs=1.f/(float)stride;
    int base=0;
    for(int j=0,mine=warp;;++j){
        const int k0=s0+2*j,k1=e0+2*j;
        const unsigned m0=__ballot_sync(0xffffffffu,k0<e0),m1=__ballot_sync(0xffffffffu,k1<e1);
        if((m0|m1)==0u) break;
        const int b1=base+__popc(m0);
        if(j==mine){                                   // uniform over the warp
            mine+=nw;
            if(k0<e0) out[base+__popc(m0&below)]=pair_entry(k0,k0+1<e0,c0,stride,rs,run);
            if(k1<e1) out[b1+__popc(m1&below)]=pair_entry(k1,k1+1<e1,c1,stride,rs,run);}
        base=b1+__popc(m1);}
    return base;
}

// G[k] = sum_n s(n) d_k w(n) over the 27 stencil nodes, for a tile s[3][TILE_S]. The weights
// are separable, w = wx wy wz: the z sums of wz s and dwz s come first, then each (x, y)
// pair adds them with dwx wy, wx dwy and wx wy.
template<class T> __device__ __forceinline__ void gather_grad(const Stencil<T>& st,const T (*s)[TILE_S],C3<T> (&G)[3])
{
#pragma unroll
    for(int k=0;k<3;++k) G[k]=c3<T>(T(0),T(0),T(0));
    const int tb=tile_addr(st.r[0]-1,st.r[1]-1,st.r[2]-1);
#pragma unroll
    for(int ox=0;ox<3;++ox)
#pragma unroll
    for(int oy=0;oy<3;++oy){
        C3<T> t,u;
#pragma unroll
        for(int oz=0;oz<3;++oz){
            const int n=tb+tile_addr(ox,oy,oz);
            const C3<T> v=c3<T>(s[0][n],s[1][n],s[2][n]);
            t=oz==0?mul(v,st.w[2][oz]):madd(v,st.w[2][oz],t);
            u=oz==0?mul(v,st.dw[2][oz]):madd(v,st.dw[2][oz],u);}
        const T dxy=st.dw[0][ox]*st.w[1][oy],xdy=st.w[0][ox]*st.dw[1][oy],wxy=st.w[0][ox]*st.w[1][oy];
        G[0]=madd(t,dxy,G[0]);G[1]=madd(t,xdy,G[1]);G[2]=madd(u,wxy,G[2]);}
}

// Conflict-free rounds for a warp's scatter into its private tile. Lanes whose particles
// share a cell are spread over successive rounds, so inside a round the lanes' cells
// differ and, for any one stencil offset, so do their nodes: one offset's read-add-write
// is conflict free. Two lanes can still reach the same node through different offsets,
// so each offset's update is ordered before the next one's with __syncwarp over the
// round's lanes. (This replaced shared-memory float atomics on one CTA-wide tile: C1's
// P2G went from ~0.2 to 0.11 ms per launch.)
struct ScatterRounds {
    int rank,rounds;
    __device__ __forceinline__ ScatterRounds(bool valid,unsigned cell)
    {
        const unsigned peers=__match_any_sync(0xffffffffu,valid?cell:(64u+(threadIdx.x&31)));
        rank=__popc(peers&lane_bits_below());
        rounds=(int)__reduce_max_sync(0xffffffffu,(unsigned)rank)+1;
    }
};

// Plasticity and transfer data of the particle in old slot src, for position i of the new buffer
// (cell `cell` of block b): the state, the cache and its identity are written there.
// Returned: stencil coordinates, HessianData, mass and velocity.
template<class T> struct Transferred { T x[3],m,V[3];HessianData<T> h; };
template<class P> __device__ __forceinline__ void update_particle(const DevState<typename P::T>& S,const SceneDev<typename P::T>& sc,const int* b,unsigned cell,
    int src,long long i,Transferred<typename P::T>& o)
{
    using T=typename P::T; using TS=typename P::TS;
    const long long pc=S.pcap;
    const T* Pin=S.pcur;T* Pout=S.pnxt;
    T F[9],X[3];
#pragma unroll
    for(int a=0;a<3;++a){X[a]=Pin[(FX+a)*pc+src];o.V[a]=Pin[(FV+a)*pc+src];}
#pragma unroll
    for(int k=0;k<9;++k) F[k]=Pin[(FF+k)*pc+src];
    T Jp=Pin[FJP*pc+src];
    o.m=Pin[FM*pc+src];
    const T V0=Pin[FV0*pc+src],lam0=Pin[FLAM0*pc+src],mu0=Pin[FMU0*pc+src];
    S.pid_nxt[i]=S.pid_cur[src];S.scn_nxt[i]=S.scn_cur[src];
#pragma unroll
    for(int a=0;a<3;++a){Pout[(FX+a)*pc+i]=X[a];Pout[(FV+a)*pc+i]=o.V[a];}
    Pout[FM*pc+i]=o.m;Pout[FV0*pc+i]=V0;Pout[FLAM0*pc+i]=lam0;Pout[FMU0*pc+i]=mu0;
    stencil_coord(sc,b,cell,X,o.x);
    if(sc.eos){
        // EOS fluid (MPM_Example.cpp:737-738): no constitutive update; the density is the Jp
        // slot. The CG's coefficient V0 k gamma rho^(gamma-1), the explicit V0/rho k rho^(gamma-1).
        const T pw=tpow(Jp,sc.eos_gamma-T(1));
        o.h=HessianData<T>{{V0/Jp*sc.bulk*pw,T(0),T(0),T(0),T(0),T(0)},T(0),V0*sc.bulk*sc.eos_gamma*pw,T(0)};}
    else{
        T R[9],lam,mu,Je;
        precompute<T,TS>(F,Jp,lam0,mu0,sc.plastic,sc.hardening,sc.cy,sc.sy,sc.hmax,R,lam,mu,Je);
        hessian_data(F,R,lam,mu,Je,V0,o.h);}
#pragma unroll
    for(int k=0;k<9;++k) Pout[(FF+k)*pc+i]=F[k];
    Pout[FJP*pc+i]=Jp;
    S.cache[i]=V4<T>{o.x[0],o.x[1],o.x[2],o.h.c1};
    S.cache[pc+i]=V4<T>{o.h.E[0],o.h.E[1],o.h.E[2],o.h.E[3]};
    S.cache[2*pc+i]=V4<T>{o.h.E[4],o.h.E[5],o.h.c2,o.h.c3};
    if constexpr(sizeof(T)==8){
        const T Sm[6]={T(1)+o.h.E[0],o.h.E[1],o.h.E[2],T(1)+o.h.E[3],o.h.E[4],T(1)+o.h.E[5]};
        T Ki[6];skew_system_inverse(Sm,Ki);
        S.cache[3*pc+i]=V4<T>{Ki[0],Ki[1],Ki[2],Ki[3]};
        S.cache[4*pc+i]=V4<T>{Ki[4],Ki[5],T(0),T(0)};}
    else S.cache[3*pc+i]=V4<T>{o.m,o.V[0],o.V[1],o.V[2]};
}

// FP64: one pass of a work item's particles through P2G. Pass qi gives lane L the cell-ordered
// particle L*stride + qi (item position inv[k] in the sorted order, read through the sort
// permutation from the old buffer), which is stored at position run[qi] + L of the new
// buffer, then scattered (m, m v and f; gravity enters in the grid update) into the warp's
// tile in rounds of lanes in distinct cells. Called by every lane of the warp.
__device__ __forceinline__ void p2g_pass(const DevState<double>& S,const SceneDev<double>& sc,const ChunkInfo<double>& ci,const int* run,
    const unsigned short* inv,const unsigned char* cellv,int qi,int stride,int np,double (*tile)[TILE_S])
{
    using T=double;
    const int k=(int)(threadIdx.x&31)*stride+qi;
    const bool valid=k<np;
    T A[6];
    Transferred<T> o;
    Stencil<T> st;
    unsigned cell=0;
    if(valid){
        const int jj=inv[k];
        const long long i=ci.s+run[qi]+(int)(threadIdx.x&31);
        cell=cellv[jj];
        update_particle<PrecFP64>(S,sc,ci.b,cell,S.perm[ci.s+jj],i,o);
        S.keys[i]=((unsigned)ci.gb<<6)|cell;
        transfer_stress(o.h,sc.eos!=0,A);
        stencil_from_coord(sc,cell,o.x,st);}
    const ScatterRounds R(valid,cell);
    for(int r=0;r<R.rounds;++r){
        const unsigned rmask=__ballot_sync(0xffffffffu,valid&&R.rank==r);
        if(valid&&R.rank==r){
            const int tb=tile_addr(st.r[0]-1,st.r[1]-1,st.r[2]-1);
#pragma unroll
            for(int k=0;k<3;++k){opaque(st.w[0][k]);opaque(st.dw[0][k]);}
            const T mv0=o.m*o.V[0],mv1=o.m*o.V[1],mv2=o.m*o.V[2];
#pragma unroll
            for(int ox=0;ox<3;++ox)
#pragma unroll
            for(int oy=0;oy<3;++oy){
                // at this (x, y): w = wxy wz and f_a = -sum_k A_ak grad_k w = -(al_a wz + be_a dwz)
                const T dxy=st.dw[0][ox]*st.w[1][oy],xdy=st.w[0][ox]*st.dw[1][oy],wxy=st.w[0][ox]*st.w[1][oy];
                const T cm=o.m*wxy,cv0=mv0*wxy,cv1=mv1*wxy,cv2=mv2*wxy;
                const T al0=-(A[0]*dxy+A[1]*xdy),al1=-(A[1]*dxy+A[3]*xdy),al2=-(A[2]*dxy+A[4]*xdy);
                const T be0=A[2]*wxy,be1=A[4]*wxy,be2=A[5]*wxy;
#pragma unroll
                for(int oz=0;oz<3;++oz){
                    const T wz=st.w[2][oz],dz=st.dw[2][oz];
                    const int t=tb+tile_addr(ox,oy,oz);
                    tile[0][t]=tfma(cm,wz,tile[0][t]);
                    tile[1][t]=tfma(cv0,wz,tile[1][t]);tile[2][t]=tfma(cv1,wz,tile[2][t]);tile[3][t]=tfma(cv2,wz,tile[3][t]);
                    tile[4][t]=tfma(-be0,dz,tfma(al0,wz,tile[4][t]));
                    tile[5][t]=tfma(-be1,dz,tfma(al1,wz,tile[5][t]));
                    tile[6][t]=tfma(-be2,dz,tfma(al2,wz,tile[6][t]));
                    __syncwarp(rmask);}}}
        __syncwarp();}
}

// The flush of a warp's (or the CTA's summed) P2G tile: one vector atomic per touched node
// and channel group.
template<class T> __device__ __forceinline__ void p2g_flush_node(const DevState<T>& S,const int* nbr,int t,const T* v)
{
    if(v[0]==T(0)&&v[4]==T(0)&&v[5]==T(0)&&v[6]==T(0)) return;
    const long long node=tile_node(nbr,t);
    if(node<0){atomicOr(&S.ctr->error,ERR_CAPACITY);return;}
    atomic_add_v3(S.gv+node,v[1],v[2],v[3],v[0]);
    atomic_add_v3(S.gf+node,v[4],v[5],v[6],T(0));
}
// Removed particles (slots >= n_valid after the sort) are carried to the new buffer as is.
template<class T> __device__ __forceinline__ void p2g_copy_removed(const DevState<T>& S,unsigned nv)
{
    const long long pc=S.pcap;
    for(long long i=(long long)nv+blockIdx.x*(long long)blockDim.x+threadIdx.x;i<S.n_total;i+=(long long)gridDim.x*blockDim.x){
        const int src=S.perm[i];
        for(int k=0;k<NB_FIELDS;++k) S.pnxt[k*pc+i]=S.pcur[k*pc+src];
        S.pid_nxt[i]=S.pid_cur[src];S.scn_nxt[i]=S.scn_cur[src];}
}

// The record of a work item, by one warp (lanes 0..31); `pairs` the length of its pair table.
template<class T> __device__ __forceinline__ void write_item(const DevState<T>& S,long long c,const ChunkInfo<T>& ci,const int* nbr,int np,int pairs)
{
    const int lane=threadIdx.x&31;
    S.items[c*ITEM_WORDS+lane]=lane==ITEM_START?ci.s:lane==ITEM_COUNT?np:lane==ITEM_SCENE?ci.scene:lane==ITEM_PAIRS?pairs:
                               lane-ITEM_NBR<27?nbr[lane-ITEM_NBR]:-1;
}
// FP64: plasticity and scatter in one kernel, a CTA per work item. The four warps sort the
// item's particles by cell together, take its passes in turn into their own tiles, and the
// tiles are summed at the flush.
template<int MINB> __global__ void __launch_bounds__(XFER_THREADS,MINB) k_p2g(DevState<double> S)
{
    pdl_enter();
    using T=double;
    constexpr int NW=XFER_THREADS/32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T (*acc)[7][TILE_S]=reinterpret_cast<T (*)[7][TILE_S]>(smem_raw);   // [warp][channel][node]
    int (*ocnt)[64]=reinterpret_cast<int (*)[64]>(smem_raw+p2g_tile_bytes<T>());
    int* rank_end=reinterpret_cast<int*>(ocnt+NW);
    unsigned short* inv=reinterpret_cast<unsigned short*>(rank_end+64);
    unsigned short* loc=inv+S.chunk;
    unsigned char* cellv=reinterpret_cast<unsigned char*>(loc+S.chunk);
    __shared__ unsigned char crank[64];
    __shared__ int nbr[27];
    __shared__ int run[129];
    const int warp=threadIdx.x>>5;
    const unsigned nc=min(S.ctr->n_chunks,(unsigned)S.chunk_cap),nv=S.ctr->n_valid;
    if(threadIdx.x<64) crank[threadIdx.x]=cell_ranks.rank[threadIdx.x];   // read after the next barrier
    for(long long c=blockIdx.x;c<nc;c+=gridDim.x){
        ChunkInfo<T> ci;
        load_chunk(S,c,nc,nv,ci,nbr);
        const int np=ci.e-ci.s,stride=(np+31)>>5;
        // a work item longer than `chunk` only arises when the work-item capacity was exceeded;
        // an empty record keeps the later kernels off it
        const bool over=np>S.chunk;
        if(warp==0){__syncwarp();write_item(S,c,ci,nbr,over?0:np,0);}
        if(over){if(threadIdx.x==0) atomicOr(&S.ctr->error,ERR_CAPACITY);continue;}   // uniform
        if(warp==0) chunk_runs(np,stride,run);        // read after the barriers in chunk_cell_order
        for(int t=threadIdx.x;t<NW*7*TILE_S;t+=blockDim.x) (&acc[0][0][0])[t]=T(0);
        chunk_cell_order(S.keys,ci.s,np,crank,ocnt,inv,loc,cellv,rank_end);
        const SceneDev<T>& sc=S.scenes[ci.scene];
        for(int qi=warp;qi<stride;qi+=NW) p2g_pass(S,sc,ci,run,inv,cellv,qi,stride,np,acc[warp]);
        __syncthreads();
        for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){
            const int ta=tile_addr(t);
            T v[7];
#pragma unroll
            for(int ch=0;ch<7;++ch){T a=T(0);
#pragma unroll
                for(int w=0;w<NW;++w) a+=acc[w][ch][ta];
                v[ch]=a;}
            p2g_flush_node(S,nbr,t,v);}
        __syncthreads();
    }
    p2g_copy_removed(S,nv);
}

// FP32, the particle part of P2G: one thread per position of the new buffer (k_items ordered
// them). Apart from the scatter it needs no shared memory, spreads a small scene's particles
// over all SMs and keeps the plasticity's code out of the scatter's loop, where the two
// together overran the instruction cache (38 % of the stall cycles on yielding particles).
// Ordering, particles and scatter against the one kernel before: 0.71 -> 0.50 ms (1.94M particles,
// 81 % yielding), 2.15 -> 1.75 ms (64-scene batch), 82 -> 62 us (60K), 2.78 -> 2.74 ms
// (21.5M unstrained particles). Bound by instruction issue where particles yield, else by HBM.
template<class P> __global__ void __launch_bounds__(XFER_THREADS,4) k_particles(DevState<typename P::T> S)
{
    pdl_enter();
    using T=typename P::T;
    const long long nv=S.ctr->n_valid;
    for(long long i=blockIdx.x*(long long)blockDim.x+threadIdx.x;i<nv;i+=(long long)gridDim.x*blockDim.x){
        const int src=S.src[i];
        const unsigned key=S.keys[i];
        const SceneDev<T>& sc=S.scenes[S.scn_cur[src]];
        int b[3];block_coords(sc,(long long)(key>>6),b);
        Transferred<T> o;
        update_particle<P>(S,sc,b,key&63u,src,i,o);}
    p2g_copy_removed(S,(unsigned)nv);
}

// Full permutation of the particle state (first grid build, before any P2G).
template<class T> __global__ void __launch_bounds__(256) k_permute(DevState<T> S)
{
    const long long pc=S.pcap;
    for(long long i=blockIdx.x*(long long)blockDim.x+threadIdx.x;i<S.n_total;i+=(long long)gridDim.x*blockDim.x){
        const int src=S.perm[i];
        for(int k=0;k<NB_FIELDS;++k) S.pnxt[k*pc+i]=S.pcur[k*pc+src];
        S.pid_nxt[i]=S.pid_cur[src];S.scn_nxt[i]=S.scn_cur[src];}
}

// Clears the accumulated node channels, records each scene's range in the work-item list and
// in the active-block list (SceneRange; the ranges were zeroed before the key pass) and, with
// `order` (FP32 substeps), puts each work item's particles in storage order: their old slots
// and keys by new position, the pair table and the record, and with `units` those of k_cg_solve.
template<class T> __global__ void __launch_bounds__(XFER_THREADS,10) k_items(DevState<T> S,int order,int units)
{
    pdl_enter();
    constexpr int NW=XFER_THREADS/32;
    const long long na=(long long)min(S.ctr->n_active,(unsigned)S.block_cap);
    const long long nn=na*64;
    const long long t0=blockIdx.x*(long long)blockDim.x+threadIdx.x,stride=(long long)gridDim.x*blockDim.x;
    const unsigned nc=min(S.ctr->n_chunks,(unsigned)S.chunk_cap),nv=S.ctr->n_valid;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int (*ocnt)[64]=reinterpret_cast<int (*)[64]>(smem_raw);
    int* rank_end=reinterpret_cast<int*>(ocnt+NW);
    unsigned short* inv=reinterpret_cast<unsigned short*>(rank_end+64);
    unsigned short* loc=inv+S.chunk;
    unsigned char* cellv=reinterpret_cast<unsigned char*>(loc+S.chunk);
    __shared__ unsigned char crank[64],cell_of[64];
    __shared__ int nbr[27];
    __shared__ int run[129];
    const int warp=threadIdx.x>>5;
    if(threadIdx.x<64){crank[threadIdx.x]=cell_ranks.rank[threadIdx.x];cell_of[threadIdx.x]=cell_ranks.cell[threadIdx.x];}   // read after the next barrier
    for(long long c=order?(long long)blockIdx.x:nc;c<nc;c+=gridDim.x){
        ChunkInfo<T> ci;
        load_chunk(S,c,nc,nv,ci,nbr);
        const int np=ci.e-ci.s,st=(np+31)>>5;
        // a work item longer than `chunk` only arises when the work-item capacity was exceeded:
        // it keeps its order, and an empty record keeps the later kernels off it
        if(np>S.chunk){                               // uniform
            if(threadIdx.x==0) atomicOr(&S.ctr->error,ERR_CAPACITY);
            for(int i=ci.s+threadIdx.x;i<ci.e;i+=blockDim.x) S.src[i]=S.perm[i];
            if(warp==0){__syncwarp();write_item(S,c,ci,nbr,0,0);}
            __syncthreads();
            continue;}
        if(warp==0) chunk_runs(np,st,run);            // read after the barriers in chunk_cell_order
        chunk_cell_order(S.keys,ci.s,np,crank,ocnt,inv,loc,cellv,rank_end);
        const int pairs=pair_table(rank_end,cell_of,st,run,S.pairs+ci.s);
        if(warp==0) write_item(S,c,ci,nbr,np,pairs);
        if(units&&warp==1){
            const int nu=(pairs+SOLVE_UNIT-1)/SOLVE_UNIT,lane=threadIdx.x&31;
            unsigned u0=0;
            if(lane==0) u0=atomicAdd(&S.ctr->n_units,(unsigned)nu);
            u0=__shfl_sync(0xffffffffu,u0,0);
            if(lane<nu) S.units[u0+lane]=(int)((unsigned)c<<6)|lane;}
        const float rst=1.f/(float)st;
        for(int k=threadIdx.x;k<np;k+=blockDim.x){
            const int i=ci.s+slot_position(k,st,rst,run),j=inv[k];
            S.src[i]=S.perm[ci.s+j];
            S.keys[i]=((unsigned)ci.gb<<6)|cellv[j];}
        __syncthreads();}
    const V4<T> z={T(0),T(0),T(0),T(0)};
    for(long long n=t0;n<nn;n+=stride){S.gv[n]=z;S.gf[n]=z;}
    auto chunk_scene=[&](long long c){return S.scn_cur[S.perm[S.chunk_start[c]]];};
    for(long long c=t0;c<nc;c+=stride){
        const int sc=chunk_scene(c);
        if(c==0||chunk_scene(c-1)!=sc) S.srange[sc].c0=(int)c;
        if(c+1==nc||chunk_scene(c+1)!=sc) S.srange[sc].c1=(int)(c+1);}
    for(long long b=t0;b<na;b+=stride){
        const int sc=S.active_scene[b];
        if(b==0||S.active_scene[b-1]!=sc) S.srange[sc].b0=(int)b;
        if(b+1==na||S.active_scene[b+1]!=sc) S.srange[sc].b1=(int)(b+1);}
}

// Mass-only P2G for the first-touch volumes (MPM_Driver::Initialize -> Rasterize).
template<class T> __global__ void __launch_bounds__(XFER_THREADS) k_p2g_mass(DevState<T> S)
{
    __shared__ T acc[TILE_S];
    __shared__ int nbr[27];
    const unsigned nc=min(S.ctr->n_chunks,(unsigned)S.chunk_cap),nv=S.ctr->n_valid;
    for(long long c=blockIdx.x;c<nc;c+=gridDim.x){
        ChunkInfo<T> ci;load_chunk(S,c,nc,nv,ci,nbr);
        for(int t=threadIdx.x;t<TILE_S;t+=blockDim.x) acc[t]=T(0);
        __syncthreads();
        const SceneDev<T>& sc=S.scenes[ci.scene];
        const int np=ci.e-ci.s;
        FOR_INTERLEAVED(np,j){
            const int i=ci.s+j;
            const long long pc=S.pcap;
            T X[3];for(int a=0;a<3;++a) X[a]=S.pcur[(FX+a)*pc+i];
            const T m=S.pcur[FM*pc+i];
            Stencil<T> st;make_stencil(sc,ci.b,S.keys[i],X,st);
            for(int ox=0;ox<3;++ox) for(int oy=0;oy<3;++oy) for(int oz=0;oz<3;++oz){
                const int t=tile_addr(st.r[0]+ox-1,st.r[1]+oy-1,st.r[2]+oz-1);
                atomicAdd(&acc[t],st.w[0][ox]*st.w[1][oy]*st.w[2][oz]*m);}}
        __syncthreads();
        for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){
            const int ta=tile_addr(t);
            if(acc[ta]==T(0)) continue;
            const long long node=tile_node(nbr,t);
            if(node<0){atomicOr(&S.ctr->error,ERR_CAPACITY);continue;}
            atomicAdd(&S.gv[node].w,acc[ta]);}
        __syncthreads();
    }
}
// Process_Waiting_Particles (MPM_Example.cpp:827-840): V0 = m_p/(sum_i w_ip m_i/dx^3)
// for particles whose V0 is not positive.
template<class T> __global__ void __launch_bounds__(XFER_THREADS) k_init_volume(DevState<T> S)
{
    __shared__ T tm[TILE_S];
    __shared__ int nbr[27];
    const unsigned nc=min(S.ctr->n_chunks,(unsigned)S.chunk_cap),nv=S.ctr->n_valid;
    for(long long c=blockIdx.x;c<nc;c+=gridDim.x){
        ChunkInfo<T> ci;load_chunk(S,c,nc,nv,ci,nbr);
        __syncthreads();
        for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){const long long node=tile_node(nbr,t);tm[tile_addr(t)]=node<0?T(0):S.gv[node].w;}
        __syncthreads();
        const SceneDev<T>& sc=S.scenes[ci.scene];
        for(int i=ci.s+threadIdx.x;i<ci.e;i+=blockDim.x){
            const long long pc=S.pcap;
            if(S.pcur[FV0*pc+i]>T(0)) continue;
            T X[3];for(int a=0;a<3;++a) X[a]=S.pcur[(FX+a)*pc+i];
            Stencil<T> st;make_stencil(sc,ci.b,S.keys[i],X,st);
            T density=T(0);
            for(int ox=0;ox<3;++ox) for(int oy=0;oy<3;++oy) for(int oz=0;oz<3;++oz){
                const int t=tile_addr(st.r[0]+ox-1,st.r[1]+oy-1,st.r[2]+oz-1);
                density+=st.w[0][ox]*st.w[1][oy]*st.w[2][oz]*tm[t];}
            density*=T(1)/(sc.dx[0]*sc.dx[1]*sc.dx[2]);
            S.pcur[FV0*pc+i]=S.pcur[FM*pc+i]/density;}
        __syncthreads();
    }
}

// =====================================================================================
// K4: grid update, one thread per node. Interior where m>0 (Flag_Setup_Helper.h:25-35),
// v=mv/m (Velocity_Normalization_Helper.h:39-52), v*=v+dt/m f (Explicit_Force_Helper.h:
// 43-56), plane barriers in list order (Grid_Based_Collision_Helper.h:57-85), rhs=v*
// (MPM_RHS_Helper.h:39-50), x=v*, s=0, and the CG state reset. The last CTA sets each
// scene's tolerance max(abs, rel*max|v*|).
// =====================================================================================
template<class T> __global__ void __launch_bounds__(NODE_THREADS) k_grid_update(DevState<T> S)
{
    pdl_enter();
    __shared__ SceneRed R;
    const long long nn=(long long)min(S.ctr->n_active,(unsigned)S.block_cap)*64;
    const unsigned parts=taking_part(nn,blockDim.x);
    if(blockIdx.x>=parts) return;
    red_init(R,S.n_scenes);
    __syncthreads();
    const V4<T> z={T(0),T(0),T(0),T(0)};
    for(long long n=blockIdx.x*(long long)blockDim.x+threadIdx.x;n<nn;n+=(long long)gridDim.x*blockDim.x){
        const int blk=(int)(n>>6);
        const int scene=S.active_scene[blk];
        const SceneDev<T>& sc=S.scenes[scene];
        const V4<T> a=S.gv[n];
        const T m=a.w;
        T vn=T(0);unsigned cnt=0;
        if(m>T(0)){
            const T inv=T(1)/m;
            const T v[3]={a.x*inv,a.y*inv,a.z*inv};
            const V4<T> f=S.gf[n];
            // v* = v + dt (f/m + g): gravity needs no scatter, its force at a node is m g
            const T dt=(T)(*S.dtp),c=dt/m;
            T vs[3]={v[0]+(c*f.x+dt*sc.gravity[0]),v[1]+(c*f.y+dt*sc.gravity[1]),v[2]+(c*f.z+dt*sc.gravity[2])};
            unsigned char proj=0;
            if(sc.n_barriers){
                T x[3];node_center(S,sc,n,blk,x);
                for(int b=0;b<sc.n_barriers;++b){
                    if(!inside_barrier(sc,b,x)) continue;
                    proj=(unsigned char)(sc.project!=0);
                    if(sc.bsticky[b]){vs[0]=vs[1]=vs[2]=T(0);continue;}
                    const T nx=sc.bn[b][0],ny=sc.bn[b][1],nz=sc.bn[b][2],mu=sc.bmu[b];
                    const T proj=vs[0]*nx+vs[1]*ny+vs[2]*nz;
                    if(proj<T(0)){
                        vs[0]-=nx*proj;vs[1]-=ny*proj;vs[2]-=nz*proj;
                        const T nv=mpm_sqrt(vs[0]*vs[0]+vs[1]*vs[1]+vs[2]*vs[2]);
                        if(-proj*mu<nv){const T k=proj*mu/nv;vs[0]+=vs[0]*k;vs[1]+=vs[1]*k;vs[2]+=vs[2]*k;}
                        else{vs[0]=vs[1]=vs[2]=T(0);}}}}
            S.gv[n]=V4<T>{v[0],v[1],v[2],m};
            S.gx[n]=V4<T>{vs[0],vs[1],vs[2],T(0)};
            S.gr[n]=V4<T>{vs[0],vs[1],vs[2],T(0)};
            S.gm[n]=m;S.gproj[n]=proj;
            vn=vs[0]*vs[0]+vs[1]*vs[1]+vs[2]*vs[2];cnt=1;}
        else{S.gv[n]=z;S.gx[n]=z;S.gr[n]=z;S.gm[n]=T(0);S.gproj[n]=0;}
        S.gs[n]=z;S.gf[n]=z;
        const double wmax=warp_max<double>((double)vn);
        const unsigned wc=warp_sum<unsigned>(cnt);
        if((threadIdx.x&31)==0){if(wmax>0.) atomicMax(&R.mx[scene],dbits(wmax));if(wc) atomicAdd(&R.cnt[scene],(unsigned long long)wc);}
    }
    red_finish<true>(R,S.n_scenes,S.acc2,&S.ctr->ticket[0],parts,[&](int i,double mx,unsigned long long cnt){
        const SceneDev<T>& sc=S.scenes[i];CGState& st=S.cg[i];
        st.tol=fmax(sc.cg_abs_tol,sc.cg_rel_tol*sqrt(mx));
        st.rho=0.;st.beta=0.;st.msq=0.;st.residual=0.;st.iters=0;st.done=0;st.converged=0;st.n_interior=(int)cnt;
    });
}

__device__ __forceinline__ float2 pabs(float2 a){return make_float2(fabsf(a.x),fabsf(a.y));}
// Sums with a product in them as two scalar operations: the assembler fuses a packed product
// and a packed sum of it, and the weights have to be those of bspline_weights bit for bit (a
// node that only the edge of a stencil reaches has its mass from their last bits).
__device__ __forceinline__ float2 sadd(float2 a,float2 b){return make_float2(__fadd_rn(a.x,b.x),__fadd_rn(a.y,b.y));}
__device__ __forceinline__ float2 ssub(float2 a,float2 b){return make_float2(__fsub_rn(a.x,b.x),__fsub_rn(a.y,b.y));}
// bspline_weights of two coordinates, operation for operation: the same bits.
__device__ __forceinline__ void bspline_weights2(float2 x,float2 inv_dx,float2 (&w)[3],float2 (&dw)[3])
{
    const float2 half=pdup(.5f),th=pdup(1.5f);
    w[0]=pabs(padd(ssub(pmul(pmul(half,x),x),pmul(th,x)),pdup(1.125f)));
    dw[0]=pmul(psub(x,th),inv_dx);
    float2 y=psub(x,pdup(1.f));
    w[1]=pabs(ssub(pdup(.75f),pmul(y,y)));
    dw[1]=pmul(pmul(pdup(-2.f),y),inv_dx);
    y=psub(y,pdup(1.f));
    w[2]=pabs(padd(sadd(pmul(pmul(half,y),y),pmul(th,y)),pdup(1.125f)));
    dw[2]=pmul(padd(y,th),inv_dx);
}
// =====================================================================================
// K5: Hessian action q_raw = K s for every scene still iterating (MPM_CG_System::Force,
// MPM_CG_System.h:150-215): gather dF = (sum_i s_i grad w_i^T) Fe, dP = dP/dF:dF, scatter
// (V0 Fe dP^T)^T grad w_i. The gathered vector is x (FROM_X, for r = b - A x) or the new
// search direction s = r + beta s_old, formed on the fly from r and the old s.
// =====================================================================================
// FP64: one pass of a work item gives lane L the cell-ordered particle L*stride + qi (stored
// by P2G at position run[qi] + L). It gathers G = sum_n s(n) grad w(n)^T from the staged
// vector tile sv, forms B and scatters B grad w into the warp's private tile in rounds of
// lanes in distinct cells. Called by every lane of the warp.
__device__ __forceinline__ void hessian_pass(const DevState<double>& S,const SceneDev<double>& sc,int s,const int* run,int qi,int stride,int np,
    const double (*sv)[TILE_S],double (*tile)[TILE_S],NodeSum<double>& sks)
{
    using T=double;
    const int j=(int)(threadIdx.x&31)*stride+qi;
    const bool valid=j<np;
    const int i=s+run[qi]+(int)(threadIdx.x&31);
    C3<T> B[3];
    Stencil<T> st;
    unsigned cell=0;
    if(valid){
        const long long pc=S.pcap;
        const V4<T> q0=S.cache[i],q1=S.cache[pc+i],q2=S.cache[2*pc+i],q3=S.cache[3*pc+i],q4=S.cache[4*pc+i];
        cell=S.keys[i]&63u;
        const T Sm[6]={T(1)+q1.x,q1.y,q1.z,T(1)+q1.w,q2.x,T(1)+q2.y},Ki[6]={q3.x,q3.y,q3.z,q3.w,q4.x,q4.y},x[3]={q0.x,q0.y,q0.z};
        stencil_from_coord(sc,cell,x,st);
        C3<T> G[3];
        gather_grad(st,sv,G);
        T bg;
        if(sc.eos) fluid_stress<T>(G,q2.z,B,bg);
        else hessian_stress<T>(G,Sm,q0.w,q2.z,q2.w,Ki,B,bg);
        sks.add(bg);}
    const ScatterRounds R(valid,cell);
    for(int r=0;r<R.rounds;++r){
        const unsigned rmask=__ballot_sync(0xffffffffu,valid&&R.rank==r);
        if(valid&&R.rank==r){
            const int tb=tile_addr(st.r[0]-1,st.r[1]-1,st.r[2]-1);
#pragma unroll
            for(int ox=0;ox<3;++ox)
#pragma unroll
            for(int oy=0;oy<3;++oy){
                // q = sum_k B_k grad_k w = al wz + be dwz at this (x, y)
                const C3<T> al=madd(B[1],st.w[0][ox]*st.dw[1][oy],mul(B[0],st.dw[0][ox]*st.w[1][oy]));
                const C3<T> be=mul(B[2],st.w[0][ox]*st.w[1][oy]);
#pragma unroll
                for(int oz=0;oz<3;++oz){
                    const int t=tb+tile_addr(ox,oy,oz);
                    const C3<T> q=madd(be,st.dw[2][oz],madd(al,st.w[2][oz],c3<T>(tile[0][t],tile[1][t],tile[2][t])));
                    tile[0][t]=cx(q);tile[1][t]=cy(q);tile[2][t]=q.z;
                    __syncwarp(rmask);}}}
        __syncwarp();}
}

// The FP32 products: two particles of one cell per lane (the pair table), every operation on both as a
// packed pair: (p, q) of the two particles in one register pair, each half rounded like the
// scalar operation. The 81 node values of the cell's stencil are read once for both, and
// both particles' forces are added to the tile in one read and one write per node. The
// particles' vectors arrive in shared memory by asynchronous copies issued one pass ahead
// (slots[k][lane], read only by the lane that copied them), so that no load latency is
// left in a pass and the coefficients take no registers during the gather.
// Bound by the FMA pipe and issue (53 % each busy, 4 CTAs per SM): per product 0.158 ->
// 0.107 ms on 1.94M particles, 1.32 -> 0.83 ms on 21.5M, against one particle per lane with
// its Fe, Re, lambda, mu and V0 read as 25 separate words. Of that the stress form of
// HessianData gives 1.32 -> 1.08, pairs, item records and copies ahead the rest.
// The first N cache vectors of a pair's particles into slots[N*h + k][lane].
template<int N> __device__ __forceinline__ void copy_pair(const DevState<float>& S,int s,unsigned entry,V4<float> (*slots)[32])
{
    const int lane=threadIdx.x&31;
#pragma unroll
    for(int h=0;h<2;++h){
        const V4<float>* p=S.cache+s+((entry>>(12*h))&4095u);
#pragma unroll
        for(int k=0;k<N;++k){
            const unsigned d=(unsigned)__cvta_generic_to_shared(&slots[N*h+k][lane]);
            asm volatile("cp.async.cg.shared.global [%0],[%1],16;"::"r"(d),"l"(p+k*S.pcap):"memory");}}
}
// A single pass that a warp runs again and again (k_cg_solve): once copied, its pairs stay in
// the warp's slots and its entry here.
struct PairPass { unsigned entry=0u; bool ready=false; };
// The passes m0, m0 + dm, ... (pair index of the pass's first lane) of a work item of M pairs.
__device__ __forceinline__ void hessian_pairs(const DevState<float>& S,const SceneDev<float>& sc,int s,int M,int m0,int dm,
    const float (*sv)[TILE_S],float (*tile)[TILE_S],V4<float> (*slots)[32],NodeSum<float>& sks,
    PairPass& pass)
{
    const unsigned* tab=S.pairs+s;
    const int lane=threadIdx.x&31;
    unsigned entry=pass.entry,next=0;
    if(!pass.ready&&m0+lane<M){entry=tab[m0+lane];copy_pair<3>(S,s,entry,slots);}
    pass.entry=entry;pass.ready=m0+dm>=M;
    if(m0+dm+lane<M) next=tab[m0+dm+lane];
    for(int m=m0;m<M;m+=dm){
        const bool valid=m+lane<M;
        const unsigned cell=(entry>>24)&63u;
        const int tb=tile_addr((int)(cell&3u),(int)((cell>>2)&3u),(int)(cell>>4));
        float2 B[3][3],w[3][3],dw[3][3];      // B[component][direction], w[axis][node]
        asm volatile("cp.async.wait_all;":::"memory");
        // formed before the gather and again before the scatter: kept across the stress the
        // 36 registers would cost a resident CTA
        auto weights=[&](float2 (&w)[3][3],float2 (&dw)[3][3]){
            const volatile V4<float>* p=&slots[0][lane];const volatile V4<float>* q=&slots[3][lane];
            bspline_weights2(make_float2(p->x,q->x),pdup(sc.inv_dx[0]),w[0],dw[0]);
            bspline_weights2(make_float2(p->y,q->y),pdup(sc.inv_dx[1]),w[1],dw[1]);
            bspline_weights2(make_float2(p->z,q->z),pdup(sc.inv_dx[2]),w[2],dw[2]);};
        if(valid){
            weights(w,dw);
            float2 G[3][3];
#pragma unroll
            for(int ox=0;ox<3;++ox)
#pragma unroll
            for(int oy=0;oy<3;++oy){
                const float2 dxy=pmul(dw[0][ox],w[1][oy]),xdy=pmul(w[0][ox],dw[1][oy]),wxy=pmul(w[0][ox],w[1][oy]);
#pragma unroll
                for(int a=0;a<3;++a){
                    float2 t,u;
#pragma unroll
                    for(int oz=0;oz<3;++oz){
                        const float2 v=pdup(sv[a][tb+tile_addr(ox,oy,oz)]);
                        t=oz==0?pmul(v,w[2][oz]):pfma(v,w[2][oz],t);
                        u=oz==0?pmul(v,dw[2][oz]):pfma(v,dw[2][oz],u);}
                    const bool first=ox==0&&oy==0;
                    G[a][0]=first?pmul(t,dxy):pfma(t,dxy,G[a][0]);
                    G[a][1]=first?pmul(t,xdy):pfma(t,xdy,G[a][1]);
                    G[a][2]=first?pmul(u,wxy):pfma(u,wxy,G[a][2]);}}
            const V4<float> p2=slots[2][lane],q2=slots[5][lane];
            const bool two=(entry&PAIR_TWO)!=0u;                    // no second particle: no force
            const float2 c2=make_float2(p2.z,two?q2.z:0.f);
            float2 bg;
            if(sc.eos) fluid_stress2(G,c2,B,bg);                    // uniform
            else{
                const V4<float> p1=slots[1][lane],q1=slots[4][lane];
                const float2 one=pdup(1.f);
                const float2 Sm[6]={padd(one,make_float2(p1.x,q1.x)),make_float2(p1.y,q1.y),make_float2(p1.z,q1.z),
                                    padd(one,make_float2(p1.w,q1.w)),make_float2(p2.x,q2.x),padd(one,make_float2(p2.y,q2.y))};
                hessian_stress2(G,Sm,make_float2(slots[0][lane].w,two?slots[3][lane].w:0.f),c2,make_float2(p2.w,two?q2.w:0.f),B,bg);}
            sks.add(bg.x+bg.y);
            weights(w,dw);}
        entry=next;
        if(m+dm+lane<M) copy_pair<3>(S,s,entry,slots);
        if(m+2*dm+lane<M) next=tab[m+2*dm+lane];
        const ScatterRounds R(valid,cell);
        for(int r=0;r<R.rounds;++r){
            const unsigned rmask=__ballot_sync(0xffffffffu,valid&&R.rank==r);
            if(valid&&R.rank==r){
#pragma unroll
                for(int k=0;k<3;++k){
                    opaque(w[0][k]);opaque(dw[0][k]);
#pragma unroll
                    for(int a=0;a<3;++a) opaque(B[a][k]);}
#pragma unroll
                for(int ox=0;ox<3;++ox)
#pragma unroll
                for(int oy=0;oy<3;++oy){
                    const float2 dxy=pmul(dw[0][ox],w[1][oy]),xdy=pmul(w[0][ox],dw[1][oy]),wxy=pmul(w[0][ox],w[1][oy]);
                    float2 al[3],be[3];
#pragma unroll
                    for(int a=0;a<3;++a){al[a]=pfma(B[a][1],xdy,pmul(B[a][0],dxy));be[a]=pmul(B[a][2],wxy);}
#pragma unroll
                    for(int oz=0;oz<3;++oz){
                        const int t=tb+tile_addr(ox,oy,oz);
                        float v[3];
#pragma unroll
                        for(int a=0;a<3;++a){
                            const float2 f=pfma(be[a],dw[2][oz],pfma(al[a],w[2][oz],make_float2(tile[a][t],0.f)));
                            v[a]=f.x+f.y;}
#pragma unroll
                        for(int a=0;a<3;++a) tile[a][t]=v[a];
                        __syncwarp(rmask);}}}
            __syncwarp();}
    }
}

// The Hessian's two ways of taking work items, one kernel (the form is a launch argument,
// uniform over the grid):
// - CTA per item (HESS_CTA): the CTA's warps share one staged vector tile and take the
//   passes of the item in turn, each into its own accumulation tile; the tiles are summed
//   at the flush. Suits launches with few work items (one scene, or the last CG trips of a
//   batch, where one scene still iterates).
// - Warp per item (HESS_WARP): each warp takes whole work items on its own, with its own
//   staged vector and accumulation tiles, synchronised by __syncwarp only (no CTA barrier
//   inside the loop). Suits launches with many items per SM (the 64-scene batch: about
//   37,000); with few, one warp per item leaves SMs idle.
// - HESS_AUTO: per launch, a warp per item when the launch has at least as many work items
//   as warps can be resident (`warp_min`, set by the host from the SM count and the
//   occupancy variant), else a CTA per item (the count is known on the device: all items
//   for the first product, the iterating scenes' items for a loop trip).
constexpr int HESS_CTA=0, HESS_WARP=1, HESS_AUTO=2;
// Shared memory of one warp: accumulated tile, staged tile and, in FP32, the copied pairs.
template<class T> __host__ __device__ constexpr int hess_warp_bytes(){return 6*TILE_S*(int)sizeof(T)+(sizeof(T)==4?6*32*16:0);}
template<class T> constexpr int hess_kernel_smem_bytes(){return (XFER_THREADS/32)*hess_warp_bytes<T>();}
// Tile node t packed as neighbour index (5 bits), local node (6 bits), tile address.
__device__ __forceinline__ unsigned tile_map_entry(int t)
{
    const int tx=t%TILE,ty=(t/TILE)%TILE,tz=t/(TILE*TILE);
    const int idx=(tx+3)/4+3*((ty+3)/4)+9*((tz+3)/4),l=((tx+3)&3)|(((ty+3)&3)<<2)|(((tz+3)&3)<<4);
    return (unsigned)idx|((unsigned)l<<5)|((unsigned)tile_addr(t)<<11);
}
// The products scale the gathered vector by the power of two below dt: G, and with it B, K s and
// s^T K s, then have the magnitudes that dt^2 K has beside the masses, in range where a stiff
// material's own are not (at 6e25 Pa and 1e10 m/s FP32 overflows in s^T K s). The scaling is
// exact: no bit changes where nothing leaves the range.
template<class T> struct ProductScale {
    T scale;       // of the gathered vector, so of K s in the grid; s^T K s has its square
    T kdt;         // dt^2/scale, for K s
    T sks;         // dt^2/scale^2, for s^T K s
    __device__ __forceinline__ explicit ProductScale(T dt)
    {
        T inv;
        if constexpr(sizeof(T)==4){
            const int e=min(max(__float_as_int(dt)&0x7f800000,0x00800000),0x7e800000);
            scale=__int_as_float(e);inv=__int_as_float(0x7f000000-e);}
        else{
            const int e=min(max(__double2hiint(dt)&0x7ff00000,0x00100000),0x7fd00000);
            scale=__hiloint2double(e,0);inv=__hiloint2double(0x7fe00000-e,0);}
        const T f=dt*inv;
        kdt=dt*f;sks=f*f;
    }
};
// The gathered vector at the item's tile nodes, times `scale`, by NT threads: the loads of a batch of nodes
// are all issued before one is used (a node's address needs only the item record).
template<class T,int NT> __device__ __forceinline__ void stage_vector(const DevState<T>& S,const int* nbr,const unsigned* tmap,bool from_x,
    T beta,T scale,T (*sv)[TILE_S],int tid)
{
    constexpr int IT=(TILE_N+NT-1)/NT,BATCH=sizeof(T)==8?1:IT;
#pragma unroll
    for(int i0=0;i0<IT;i0+=BATCH){
        V4<T> a[BATCH],b[BATCH];unsigned ta[BATCH];
#pragma unroll
        for(int i=0;i<BATCH;++i){
            const int t=tid+(i0+i)*NT;
            a[i]=b[i]=V4<T>{T(0),T(0),T(0),T(0)};ta[i]=~0u;
            if(t<TILE_N){
                const unsigned e=tmap[t];
                ta[i]=e>>11;
                const int blk=nbr[e&31u];
                if(blk>=0){
                    const long long node=(long long)blk*64+((e>>5)&63u);
                    if(from_x) a[i]=S.gx[node];
                    else{a[i]=S.gr[node];b[i]=S.gs[node];}}}}
#pragma unroll
        for(int i=0;i<BATCH;++i) if(ta[i]!=~0u){
            sv[0][ta[i]]=scale*(from_x?a[i].x:a[i].x+beta*b[i].x);
            sv[1][ta[i]]=scale*(from_x?a[i].y:a[i].y+beta*b[i].y);
            sv[2][ta[i]]=scale*(from_x?a[i].z:a[i].z+beta*b[i].z);}}
}
// Adds an item's sum at a tile node to the grid.
template<class T> __device__ __forceinline__ void add_tile_node(const DevState<T>& S,const int* rec,unsigned e,T v0,T v1,T v2)
{
    if(v0==T(0)&&v1==T(0)&&v2==T(0)) return;
    const int blk=rec[ITEM_NBR+(e&31u)];
    if(blk>=0) atomic_add_v3(S.gf+(long long)blk*64+((e>>5)&63u),v0,v1,v2,T(0));
}
template<class P,bool FROM_X,int MINB> __global__ void __launch_bounds__(XFER_THREADS,MINB) k_hessian(DevState<typename P::T> S,int form,long long warp_min)
{
    pdl_enter();
    using T=typename P::T;
    constexpr int NW=XFER_THREADS/32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int rec_s[NW][ITEM_WORDS];
    __shared__ int run_s[sizeof(T)==8?NW:1][129];
    __shared__ unsigned tmap[TILE_N];
    __shared__ ListSmem lsm;
    __shared__ T scale;                            // a register of it would make the product spill
    const int warp=threadIdx.x>>5,lane=threadIdx.x&31;
    // the first product (FROM_X) covers every work item; a loop trip only the work items of
    // the scenes still iterating (the list the previous convergence check wrote)
    const long long nwork=FROM_X?(long long)min(S.ctr->n_chunks,(unsigned)S.chunk_cap):S.alist->cpre[S.alist->n];
    if(form==HESS_AUTO) form=nwork>=warp_min?HESS_WARP:HESS_CTA;
    if((form==HESS_CTA?(long long)blockIdx.x:(long long)blockIdx.x*NW)>=nwork) return;     // no item for this CTA
    auto tile_of=[&](int w){return reinterpret_cast<T (*)[TILE_S]>(smem_raw+w*hess_warp_bytes<T>());};   // [component][node]
    T (*q)[TILE_S]=tile_of(warp);                  // accumulated
    V4<float> (*slots)[32]=reinterpret_cast<V4<float> (*)[32]>(smem_raw+warp*hess_warp_bytes<T>()+6*TILE_S*sizeof(T));
    for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x) tmap[t]=tile_map_entry(t);
    for(int t=lane;t<3*TILE_S;t+=32) (&q[0][0])[t]=T(0);
    if(threadIdx.x==0) scale=ProductScale<T>((T)(*S.dtp)).scale;
    if(!FROM_X) load_active_list(S.alist,lsm,false);
    __syncthreads();
    auto item=[&](long long w){
        if(FROM_X) return w;
        const int j=list_find(lsm,(int)w);return S.srange[lsm.scene[j]].c0+(w-lsm.pre[j]);};
    // s^T K s of a loop trip (k_cg_update), per lane until the warp's scene changes
    NodeSum<T> sks;int sks_scene=-1;
    auto add_sks=[&](int next){
        if(!FROM_X&&sks_scene>=0&&sks_scene!=next){
            const double v=warp_value(sks);
            if(lane==0&&v!=0.) atomicAdd(&S.acc[sks_scene].sks,v);
            sks=NodeSum<T>();}
        sks_scene=next;};
    // the passes of an item: pairs (FP32) or cell-ordered particles (FP64), `first` of every `of`
    auto passes=[&](const SceneDev<T>& sc,const int* rec,const T (*sv)[TILE_S],int* run,int first,int of){
        if constexpr(sizeof(T)==4){PairPass pass;hessian_pairs(S,sc,rec[ITEM_START],rec[ITEM_PAIRS],first*32,of*32,sv,q,slots,sks,pass);}
        else{
            const int np=rec[ITEM_COUNT],stride=(np+31)>>5;
            for(int qi=first;qi<stride;qi+=of) hessian_pass(S,sc,rec[ITEM_START],run,qi,stride,np,sv,q,sks);}};
    if(form==HESS_CTA){
        T (*sv)[TILE_S]=tile_of(0)+3;
        int* rec=rec_s[0];int* run=run_s[0];
        int mine=blockIdx.x<nwork?S.items[item(blockIdx.x)*ITEM_WORDS+lane]:0;
        for(long long w=blockIdx.x;w<nwork;w+=gridDim.x){
            if(warp==0) rec[lane]=mine;
            __syncthreads();
            if(w+gridDim.x<nwork) mine=S.items[item(w+gridDim.x)*ITEM_WORDS+lane];
            const int scene=rec[ITEM_SCENE];
            stage_vector<T,XFER_THREADS>(S,rec+ITEM_NBR,tmap,FROM_X,FROM_X?T(0):(T)S.cg[scene].beta,scale,sv,threadIdx.x);
            if constexpr(sizeof(T)==8) if(warp==0) chunk_runs(rec[ITEM_COUNT],(rec[ITEM_COUNT]+31)>>5,run);
            __syncthreads();
            add_sks(scene);
            passes(S.scenes[scene],rec,sv,run,warp,NW);
            __syncthreads();
            for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){
                const unsigned e=tmap[t];
                T v[3];
#pragma unroll
                for(int ch=0;ch<3;++ch){T a=T(0);
#pragma unroll
                    for(int w2=0;w2<NW;++w2){T* p=&tile_of(w2)[ch][e>>11];a+=*p;*p=T(0);}
                    v[ch]=a;}
                add_tile_node(S,rec,e,v[0],v[1],v[2]);}
            __syncthreads();
        }
    }
    else{
        T (*sv)[TILE_S]=q+3;
        int* rec=rec_s[warp];int* run=run_s[sizeof(T)==8?warp:0];
        const long long w0=(long long)blockIdx.x*NW+warp,dw=(long long)gridDim.x*NW;
        int mine=w0<nwork?S.items[item(w0)*ITEM_WORDS+lane]:0;
        for(long long w=w0;w<nwork;w+=dw){
            rec[lane]=mine;
            __syncwarp();
            if(w+dw<nwork) mine=S.items[item(w+dw)*ITEM_WORDS+lane];
            const int scene=rec[ITEM_SCENE];
            stage_vector<T,32>(S,rec+ITEM_NBR,tmap,FROM_X,FROM_X?T(0):(T)S.cg[scene].beta,scale,sv,lane);
            if constexpr(sizeof(T)==8) chunk_runs(rec[ITEM_COUNT],(rec[ITEM_COUNT]+31)>>5,run);
            __syncwarp();
            add_sks(scene);
            passes(S.scenes[scene],rec,sv,run,0,1);
            __syncwarp();
            for(int t=lane;t<TILE_N;t+=32){
                const unsigned e=tmap[t];
                T* p=&q[0][e>>11];
                const T v0=p[0],v1=p[TILE_S],v2=p[2*TILE_S];
                p[0]=p[TILE_S]=p[2*TILE_S]=T(0);
                add_tile_node(S,rec,e,v0,v1,v2);}
            __syncwarp();
        }
    }
    add_sks(-1);
}

// =====================================================================================
// K3b: the scatter of P2G in FP32 (Rasterize, MPM_Example.cpp:520-537; Apply_Explicit_Force,
// :757-784): m, m v and f = -sum_p V0 P Fe^T grad w of two particles of one cell per lane, as
// the Hessian product scatters, into the warp's 7-channel tile. The stress is formed from the
// cache that the products read. A work item is taken by a CTA, its passes split over 2 or 4
// CTAs where items are few, or by a warp where there are at least as many as resident warps.
// =====================================================================================
constexpr int P2G_CH=7;
__host__ __device__ constexpr int scatter_warp_bytes(){return P2G_CH*TILE_S*4+8*32*16;}
__device__ __forceinline__ void scatter_pairs(const DevState<float>& S,const SceneDev<float>& sc,int s,int M,int m0,int dm,float (*tile)[TILE_S],V4<float> (*slots)[32])
{
    const unsigned* tab=S.pairs+s;
    const int lane=threadIdx.x&31;
    unsigned entry=0,next=0;
    if(m0+lane<M){entry=tab[m0+lane];copy_pair<4>(S,s,entry,slots);}
    if(m0+dm+lane<M) next=tab[m0+dm+lane];
    for(int m=m0;m<M;m+=dm){
        const bool valid=m+lane<M;
        const unsigned cell=(entry>>24)&63u;
        const int tb=tile_addr((int)(cell&3u),(int)((cell>>2)&3u),(int)(cell>>4));
        float2 w[3][3],dw[3][3],mv[4],A[6];          // mv: (m, m v), A: -V0 P Fe^T
        asm volatile("cp.async.wait_all;":::"memory");
        if(valid){
            const V4<float> p0=slots[0][lane],q0=slots[4][lane],p1=slots[1][lane],q1=slots[5][lane];
            const V4<float> p2=slots[2][lane],q2=slots[6][lane],p3=slots[3][lane],q3=slots[7][lane];
            bspline_weights2(make_float2(p0.x,q0.x),pdup(sc.inv_dx[0]),w[0],dw[0]);
            bspline_weights2(make_float2(p0.y,q0.y),pdup(sc.inv_dx[1]),w[1],dw[1]);
            bspline_weights2(make_float2(p0.z,q0.z),pdup(sc.inv_dx[2]),w[2],dw[2]);
            const float on=(entry&PAIR_TWO)?1.f:0.f;   // no second particle: nothing to add
            mv[0]=make_float2(p3.x,on*q3.x);
            mv[1]=pmul(mv[0],make_float2(p3.y,q3.y));mv[2]=pmul(mv[0],make_float2(p3.z,q3.z));mv[3]=pmul(mv[0],make_float2(p3.w,q3.w));
            const float2 c1=make_float2(-p0.w,-on*q0.w),c3=make_float2(-p2.w,-on*q2.w);
            const float2 E[6]={make_float2(p1.x,q1.x),make_float2(p1.y,q1.y),make_float2(p1.z,q1.z),
                               make_float2(p1.w,q1.w),make_float2(p2.x,q2.x),make_float2(p2.y,q2.y)};
            transfer_stress2(E,c1,c3,A);
            if(sc.eos) A[0]=A[3]=A[5]=make_float2(p1.x,on*q1.x);}
        entry=next;
        if(m+dm+lane<M) copy_pair<4>(S,s,entry,slots);
        if(m+2*dm+lane<M) next=tab[m+2*dm+lane];
        const ScatterRounds R(valid,cell);
        for(int r=0;r<R.rounds;++r){
            const unsigned rmask=__ballot_sync(0xffffffffu,valid&&R.rank==r);
            if(valid&&R.rank==r){
#pragma unroll
                for(int k=0;k<3;++k){opaque(w[0][k]);opaque(dw[0][k]);}
#pragma unroll
                for(int ox=0;ox<3;++ox)
#pragma unroll
                for(int oy=0;oy<3;++oy){
                    const float2 dxy=pmul(dw[0][ox],w[1][oy]),xdy=pmul(w[0][ox],dw[1][oy]),wxy=pmul(w[0][ox],w[1][oy]);
                    float2 c[4];
#pragma unroll
                    for(int a=0;a<4;++a) c[a]=pmul(mv[a],wxy);
                    const float2 al[3]={pfma(A[1],xdy,pmul(A[0],dxy)),pfma(A[3],xdy,pmul(A[1],dxy)),pfma(A[4],xdy,pmul(A[2],dxy))};
                    const float2 be[3]={pmul(A[2],wxy),pmul(A[4],wxy),pmul(A[5],wxy)};
#pragma unroll
                    for(int oz=0;oz<3;++oz){
                        const int t=tb+tile_addr(ox,oy,oz);
                        float v[P2G_CH];
#pragma unroll
                        for(int a=0;a<4;++a){const float2 f=pfma(c[a],w[2][oz],make_float2(tile[a][t],0.f));v[a]=f.x+f.y;}
#pragma unroll
                        for(int a=0;a<3;++a){
                            const float2 f=pfma(be[a],dw[2][oz],pfma(al[a],w[2][oz],make_float2(tile[4+a][t],0.f)));
                            v[4+a]=f.x+f.y;}
#pragma unroll
                        for(int a=0;a<P2G_CH;++a) tile[a][t]=v[a];
                        __syncwarp(rmask);}}}
            __syncwarp();}
    }
}
template<int MINB> __global__ void __launch_bounds__(XFER_THREADS,MINB) k_p2g_scatter(DevState<float> S,long long warp_min)
{
    pdl_enter();
    constexpr int NW=XFER_THREADS/32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int rec_s[NW][ITEM_WORDS];
    __shared__ unsigned tmap[TILE_N];
    const int warp=threadIdx.x>>5,lane=threadIdx.x&31;
    const long long nc=min(S.ctr->n_chunks,(unsigned)S.chunk_cap),G=gridDim.x,resident=warp_min/NW;
    const bool by_warp=nc>=warp_min;
    const int split=4*nc<=resident?4:2*nc<=resident?2:1;
    const long long units=by_warp?(nc+NW-1)/NW:nc*split;
    if(blockIdx.x>=units) return;
    auto tile_of=[&](int w){return reinterpret_cast<float (*)[TILE_S]>(smem_raw+w*scatter_warp_bytes());};   // [channel][node]
    float (*tile)[TILE_S]=tile_of(warp);
    V4<float> (*slots)[32]=reinterpret_cast<V4<float> (*)[32]>(smem_raw+warp*scatter_warp_bytes()+P2G_CH*TILE_S*4);
    for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x) tmap[t]=tile_map_entry(t);
    for(int t=lane;t<P2G_CH*TILE_S;t+=32) (&tile[0][0])[t]=0.f;
    __syncthreads();
    // one vector atomic per touched node and channel group
    auto flush=[&](const int* rec,unsigned e,const float (&v)[P2G_CH]){
        if(v[0]==0.f&&v[4]==0.f&&v[5]==0.f&&v[6]==0.f) return;
        const int blk=rec[ITEM_NBR+(e&31u)];
        if(blk<0){atomicOr(&S.ctr->error,ERR_CAPACITY);return;}
        const long long node=(long long)blk*64+((e>>5)&63u);
        atomic_add_v3(S.gv+node,v[1],v[2],v[3],v[0]);
        atomic_add_v3(S.gf+node,v[4],v[5],v[6],0.f);};
    if(by_warp){
        int* rec=rec_s[warp];
        const long long w0=(long long)blockIdx.x*NW+warp,dwork=G*NW;
        int mine=w0<nc?S.items[w0*ITEM_WORDS+lane]:0;
        for(long long c=w0;c<nc;c+=dwork){
            rec[lane]=mine;
            __syncwarp();
            if(c+dwork<nc) mine=S.items[(c+dwork)*ITEM_WORDS+lane];
            scatter_pairs(S,S.scenes[rec[ITEM_SCENE]],rec[ITEM_START],rec[ITEM_PAIRS],0,32,tile,slots);
            __syncwarp();
            for(int t=lane;t<TILE_N;t+=32){
                const unsigned e=tmap[t];
                float v[P2G_CH];
#pragma unroll
                for(int ch=0;ch<P2G_CH;++ch){float* p=&tile[ch][e>>11];v[ch]=*p;*p=0.f;}
                flush(rec,e,v);}
            __syncwarp();}
        return;}
    int* rec=rec_s[0];
    for(long long u=blockIdx.x;u<units;u+=G){
        if(warp==0) rec[lane]=S.items[(u/split)*ITEM_WORDS+lane];
        __syncthreads();
        scatter_pairs(S,S.scenes[rec[ITEM_SCENE]],rec[ITEM_START],rec[ITEM_PAIRS],(warp+NW*(int)(u%split))*32,NW*split*32,tile,slots);
        __syncthreads();
        for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){
            const unsigned e=tmap[t];
            float v[P2G_CH];
#pragma unroll
            for(int ch=0;ch<P2G_CH;++ch){float a=0.f;
#pragma unroll
                for(int w2=0;w2<NW;++w2){float* p=&tile_of(w2)[ch][e>>11];a+=*p;*p=0.f;}
                v[ch]=a;}
            flush(rec,e,v);}
        __syncthreads();}
}

// r = b - (x + dt^2/m K x) on a node block, two nodes per lane, Project(r) (MPM_CG_System.h:
// 220-225, intended semantics of Project_Helper.h:30-45; the grid update flagged the nodes),
// K x cleared; <r,r>_M and max|r|^2.
template<class T> __device__ __forceinline__ void cg_start_block(const DevState<T>& S,int blk,T kdt,NodeSum<T>& rr,T& amax)
{
    T m[2];V4<T> x[2],b[2],k[2];unsigned char pj[2];
#pragma unroll
    for(int h=0;h<2;++h){const long long n=((long long)blk<<6)+h*32+(threadIdx.x&31);m[h]=S.gm[n];x[h]=S.gx[n];b[h]=S.gr[n];k[h]=S.gf[n];pj[h]=S.gproj[n];}
#pragma unroll
    for(int h=0;h<2;++h){
        const long long n=((long long)blk<<6)+h*32+(threadIdx.x&31);
        if(m[h]>T(0)){
            const T c=kdt/m[h];
            T r[3]={b[h].x-(c*k[h].x+x[h].x),b[h].y-(c*k[h].y+x[h].y),b[h].z-(c*k[h].z+x[h].z)};
            if(pj[h]) r[0]=r[1]=r[2]=T(0);
            S.gr[n]=V4<T>{r[0],r[1],r[2],T(0)};
            rr.add(r[0]*(r[0]*m[h])+r[1]*(r[1]*m[h])+r[2]*(r[2]*m[h]));
            const T cn=r[0]*r[0]+r[1]*r[1]+r[2]*r[2];
            amax=cn>amax?cn:amax;}
        S.gf[n]=V4<T>{T(0),T(0),T(0),T(0)};}
}
// The vector update of a loop trip (k_cg_update) on the node block that starts at node n0.
template<class T> __device__ __forceinline__ void cg_update_block(const DevState<T>& S,long long n0,T alpha,T beta,T kdt,NodeSum<T>& rr,NodeSum<T>& rs,
    NodeSum<T>& ss,T& amax)
{
    T m[2];V4<T> s[2],k[2],x[2],r[2];unsigned char pj[2];
#pragma unroll
    for(int h=0;h<2;++h){const long long n=n0+h*32+(threadIdx.x&31);m[h]=S.gm[n];s[h]=S.gs[n];k[h]=S.gf[n];x[h]=S.gx[n];r[h]=S.gr[n];pj[h]=S.gproj[n];}
#pragma unroll
    for(int h=0;h<2;++h){
        const long long n=n0+h*32+(threadIdx.x&31);
        if(m[h]>T(0)){
            const T c=kdt/m[h];
            s[h].x=r[h].x+beta*s[h].x;s[h].y=r[h].y+beta*s[h].y;s[h].z=r[h].z+beta*s[h].z;
            T q[3]={c*k[h].x+s[h].x,c*k[h].y+s[h].y,c*k[h].z+s[h].z};
            if(pj[h]) q[0]=q[1]=q[2]=T(0);
            x[h].x=alpha*s[h].x+x[h].x;x[h].y=alpha*s[h].y+x[h].y;x[h].z=alpha*s[h].z+x[h].z;
            r[h].x=-alpha*q[0]+r[h].x;r[h].y=-alpha*q[1]+r[h].y;r[h].z=-alpha*q[2]+r[h].z;
            S.gs[n]=s[h];S.gx[n]=x[h];S.gr[n]=r[h];
            rr.add(r[h].x*(r[h].x*m[h])+r[h].y*(r[h].y*m[h])+r[h].z*(r[h].z*m[h]));
            rs.add(r[h].x*(s[h].x*m[h])+r[h].y*(s[h].y*m[h])+r[h].z*(s[h].z*m[h]));
            ss.add(s[h].x*(s[h].x*m[h])+s[h].y*(s[h].y*m[h])+s[h].z*(s[h].z*m[h]));
            const T cn=r[h].x*r[h].x+r[h].y*r[h].y+r[h].z*r[h].z;
            amax=cn>amax?cn:amax;}
        S.gf[n]=V4<T>{T(0),T(0),T(0),T(0)};}
}
// CG start: cg_start_block on every block, then the first convergence check of the restated CG
// loop (iteration 0).
template<class P> __global__ void __launch_bounds__(NODE_THREADS) k_cg_start(DevState<typename P::T> S,unsigned long long cond,int use_cond)
{
    pdl_enter();
    using T=typename P::T;
    __shared__ WarpParts W;
    const int na=(int)min(S.ctr->n_active,(unsigned)S.block_cap);
    const T kdt=ProductScale<T>((T)(*S.dtp)).kdt;
    const WarpRange wr(na);
    if(blockIdx.x>=wr.parts) return;
    if((threadIdx.x&31)==0) W.scene[threadIdx.x>>5]=-1;
    int scene=-1;NodeSum<T> rr;T amax=T(0);
    auto flush=[&](int sc,bool last){flush_scene<1,T>(W,S.acc,sc,last,rr,rr,rr,amax);rr=NodeSum<T>();amax=T(0);};
    for(int blk=wr.b;blk<wr.b1;++blk){
        const int sb=S.active_scene[blk];
        if(sb!=scene){if(scene>=0) flush(scene,false);scene=sb;}
        cg_start_block(S,blk,kdt,rr,amax);}
    if(scene>=0) flush(scene,true);
    __shared__ int any;
    if(threadIdx.x==0) any=0;
    const bool last=parts_finish<1>(W,S.n_scenes,S.acc,&S.ctr->ticket[1],wr.parts,[&](int i,const double* sum,double mx){
        const SceneDev<T>& sc=S.scenes[i];CGState& st=S.cg[i];
        const double cn=sqrt(mx),rr=sum[0];
        const double eps=sizeof(T)==4?1.1920928955078125e-07:2.220446049250313e-16;
        st.residual=cn;
        if(cn<=st.tol&&(0>=sc.cg_min_iters||cn<eps)){st.done=1;st.converged=1;}
        else if(sc.cg_max_iters<=0){st.done=1;st.converged=0;atomicOr(&S.ctr->error,ERR_CG_NOT_CONVERGED);}
        else{st.rho=rr;st.beta=0.;st.msq=rr;atomicOr(&any,1);}    // the first direction is r
    });
    if(last) build_active_list(S);
    if(last&&threadIdx.x==0){
        S.ctr->any_active=any;S.ctr->loop_iters=0;
        if(use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond,any?1u:0u);}
}

// A warp's share of the node blocks of the scenes in the list: a contiguous range of list
// blocks, so that the warp meets each scene once and streams whole blocks (64 nodes, two
// per lane). next() moves to list block bw (non-decreasing) and tells whether the scene
// changed; node0 is that block's first node.
struct WarpBlocks {
    int b,b1,j=0,scene=-1;long long base=0;
    __device__ __forceinline__ explicit WarpBlocks(const WarpRange& r):b(r.b),b1(r.b1){}
    __device__ __forceinline__ bool next(const ListSmem& sm,const SceneRange* sr,int bw)
    {
        if(scene>=0&&bw<sm.pre[j+1]) return false;
        while(bw>=sm.pre[j+1]) ++j;
        scene=sm.scene[j];base=sr[scene].b0-sm.pre[j];
        return true;
    }
    __device__ __forceinline__ long long node0(int bw) const {return (base+bw)<<6;}
};
// The vector update of a loop trip, one pass over the nodes: s = r + beta s_old, q = s +
// dt^2/m K s, Project(q), x += alpha s, r -= alpha q (Interior only), K s cleared for the next
// product. alpha = <r,r>_M / <s,q>_M needs no pass of its own over the nodes: <s,q>_M =
// dt^2 s^T K s + <s,s>_M, of which the Hessian product adds up s^T K s (scaled) over the particles
// (sum of B:G) and the previous update <s,s>_M = <r,r> + 2 beta <r,s_old> + beta^2
// <s_old,s_old> (s vanishes at projected nodes). Then the convergence check: stop when
// max|r| <= tol (and iters >= min, or the norm is below epsilon) or at cg_max_iters; else beta
// = <r,r>/rho, rho = <r,r>. Bound by memory on large scenes (133 bytes a node against 200 with a
// separate q pass: 114 -> 85 us a trip on the 21.5M slab), by the latency of its chain of
// reductions on small ones (22 -> 15 us).
template<class P> __global__ void __launch_bounds__(NODE_THREADS) k_cg_update(DevState<typename P::T> S,unsigned long long cond,int use_cond,int max_trips)
{
    pdl_enter();
    using T=typename P::T;
    __shared__ WarpParts W;
    __shared__ ListSmem lsm;
    const WarpRange wr(S.alist->bpre[S.alist->n]);
    if(blockIdx.x>=wr.parts) return;
    if((threadIdx.x&31)==0) W.scene[threadIdx.x>>5]=-1;
    load_active_list(S.alist,lsm,true);     // the scenes still iterating
    WarpBlocks wb(wr);
    const ProductScale<T> ps((T)(*S.dtp));
    NodeSum<T> rr,rs,ss;T amax=T(0),alpha=T(0),beta=T(0);
    auto flush=[&](int sc,bool last){
        flush_scene<3,T>(W,S.acc,sc,last,rr,rs,ss,amax);
        rr=rs=ss=NodeSum<T>();amax=T(0);};
    for(int bw=wb.b;bw<wb.b1;++bw){
        const int prev=wb.scene;
        if(wb.next(lsm,S.srange,bw)){
            if(prev>=0) flush(prev,false);
            const CGState& st=S.cg[wb.scene];
            const double sq=(double)ps.sks*S.acc[wb.scene].sks+st.msq;
            alpha=(T)(sq!=0.?st.rho/sq:(double)FLT_MAX);beta=(T)st.beta;}
        cg_update_block(S,wb.node0(bw),alpha,beta,ps.kdt,rr,rs,ss,amax);}
    if(wb.scene>=0) flush(wb.scene,true);
    __shared__ int any;
    if(threadIdx.x==0) any=0;
    const bool last=parts_finish<3>(W,S.n_scenes,S.acc,&S.ctr->ticket[3],wr.parts,[&](int i,const double* sum,double mx){
        const SceneDev<T>& sc=S.scenes[i];CGState& st=S.cg[i];
        if(st.done) return;
        S.acc[i].sks=0.;
        st.iters+=1;
        const double cn=sqrt(mx);
        const double eps=sizeof(T)==4?1.1920928955078125e-07:2.220446049250313e-16;
        st.residual=cn;
        if(cn<=st.tol&&(st.iters>=sc.cg_min_iters||cn<eps)){st.done=1;st.converged=1;}
        else if(st.iters>=sc.cg_max_iters){st.done=1;st.converged=0;atomicOr(&S.ctr->error,ERR_CG_NOT_CONVERGED);}
        else{
            st.beta=sum[0]/st.rho;st.rho=sum[0];
            st.msq=sum[0]+st.beta*(2.*sum[1]+st.beta*sum[2]);
            atomicOr(&any,1);}
    });
    if(last) build_active_list(S);
    if(last&&threadIdx.x==0){
        S.ctr->loop_iters+=1;S.ctr->total_trips+=1;
        // every scene stops by its cg_max_iters; the trip cap is a second, global bound
        if(S.ctr->loop_iters>=max_trips) any=0;
        S.ctr->any_active=any;
        if(use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond,any?1u:0u);}
}

// =====================================================================================
// The whole CG solve of a small single scene in one cooperative kernel (FP32 storage). A loop
// trip as separate kernels costs two launches, two chains of dependent loads until a CTA
// has its work item, and two last-CTA reductions, about 25 us in which a small scene computes
// for a few. Here the CTAs stay: each keeps its work item's record (and, with one pass per
// warp, its pairs) on chip, the node blocks are spread over all warps, and the phases
// (product, vector update) are separated by grid barriers whose arrivals carry the sums.
// The particles are dealt out in units of one pass per warp where there are CTAs for all of them: a
// compressed block's item has four where most have one, and the CTA that took it kept all
// others waiting (61K particles of compressed snow 227 -> 210 us a substep, 40K 194 -> 186,
// 20K of fluid 202 -> 191).
// =====================================================================================
// One arrival per CTA, after warp 0 has run `pre`; thread 0 runs `idle` while the others arrive,
// waits for all (bounded) and runs `post`. False after the limit. A round trip to L2 or a few
// dependent FP64 operations here are time of every CTA: the poll is the acquire (a fence
// and a second read after it took 0.7 us), and what the threads do not wait for is in `idle`.
// The count of arrivals wraps (at 608 CTAs after 3.5 million CG iterations); it is never further than
// one arrival per CTA from the target, so the sign of their difference decides.
constexpr int SOLVE_SPIN_LIMIT=1<<20;
__device__ __forceinline__ unsigned load_acquire(const unsigned* p){unsigned v;asm volatile("ld.acquire.gpu.global.u32 %0,[%1];":"=r"(v):"l"(p):"memory");return v;}
template<class F0,class F1,class F2> __device__ __forceinline__ bool solve_barrier(Counters* ctr,unsigned target,F0 pre,F1 idle,F2 post,int spin_limit=SOLVE_SPIN_LIMIT)
{
    __shared__ bool ok;
    __syncthreads();
    if(threadIdx.x<32){
        pre();
        __syncwarp();
        if(threadIdx.x==0){
            __threadfence();
            atomicAdd(&ctr->solve_arrived,1u);
            idle();
            int spins=0;
            unsigned seen;
            while((int)((seen=load_acquire(&ctr->solve_arrived))-target)<0&&++spins<spin_limit) if(spins>64) __nanosleep(32);
            ok=(int)(seen-target)>=0;
            if(!ok) atomicOr(&ctr->error,ERR_GRID_WAIT);
            post();}}
    __syncthreads();
    return ok;
}
template<class P> __global__ void __launch_bounds__(XFER_THREADS,4) k_cg_solve(DevState<typename P::T> S,int max_trips)
{
    using T=typename P::T;
    static_assert(sizeof(T)==4,"pair tables are FP32 only");
    static_assert(SOLVE_UNIT==32*(XFER_THREADS/32),"a unit is one pass per warp");
    constexpr int NW=XFER_THREADS/32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int rec[ITEM_WORDS];
    __shared__ unsigned tmap[TILE_N];
    __shared__ double part[NW][4];
    __shared__ T sh_alpha,sh_beta;
    __shared__ int sh_stop;
    const int warp=threadIdx.x>>5,lane=threadIdx.x&31;
    auto tile_of=[&](int w){return reinterpret_cast<T (*)[TILE_S]>(smem_raw+w*hess_warp_bytes<T>());};
    T (*q)[TILE_S]=tile_of(warp);
    T (*sv)[TILE_S]=tile_of(0)+3;
    V4<float> (*slots)[32]=reinterpret_cast<V4<float> (*)[32]>(smem_raw+warp*hess_warp_bytes<T>()+6*TILE_S*sizeof(T));
    for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x) tmap[t]=tile_map_entry(t);
    for(int t=lane;t<3*TILE_S;t+=32) (&q[0][0])[t]=T(0);
    Counters* ctr=S.ctr;
    const int nc=(int)min(ctr->n_chunks,(unsigned)S.chunk_cap),na=(int)min(ctr->n_active,(unsigned)S.block_cap);
    // A CTA for each unit where the launch has that many: nobody waits for a compressed block.
    // The CTAs without a unit or a warp's node block would only make the barriers longer. With
    // more units than CTAs whole items, or halves or quarters of their passes, are cheaper: a
    // second unit of another item is staged and flushed again (100K particles at rest 277
    // against 255 us a substep, 900K 1,476 against 1,293).
    const unsigned U=ctr->n_units;
    const bool listed=U!=0u&&U<=gridDim.x;
    const int G=listed?(int)min(gridDim.x,max(U,((unsigned)na+NW-1u)/NW)):(int)gridDim.x;
    if((int)blockIdx.x>=G) return;
    const int split=4*nc<=G?4:2*nc<=G?2:1,units=listed?(int)U:nc*split;
    const int per=(na+G*NW-1)/(G*NW),b0=min(na,((int)blockIdx.x*NW+warp)*per),b1=min(na,b0+per);
    const SceneDev<T>& sc=S.scenes[0];
    const ProductScale<T> ps((T)(*S.dtp));
    PairPass pass;                       // the warp's resident pass, when the CTA has one unit
    int held=-1;                         // unit whose item's record is in rec
    unsigned entry=0;                    // its entry
    unsigned phase=0;                    // wraps as the count does
    auto arrived=[&]{return (phase+1u)*(unsigned)G;};
    // K v for v = x, or s = r + beta s_old with s^T K s into part[][0]
    auto product=[&](bool from_x,T beta){
        NodeSum<T> sks;
        for(int u=blockIdx.x;u<units;u+=G){
            if(u!=held){
                entry=listed?(unsigned)S.units[u]:((unsigned)(u/split)<<6)|(unsigned)(u%split);
                __syncthreads();
                if(warp==0) rec[lane]=S.items[(long long)(entry>>6)*ITEM_WORDS+lane];
                held=u;pass.ready=false;
                __syncthreads();}
            stage_vector<T,XFER_THREADS>(S,rec+ITEM_NBR,tmap,from_x,beta,ps.scale,sv,threadIdx.x);
            __syncthreads();
            const int M=rec[ITEM_PAIRS],parts=listed?(M+SOLVE_UNIT-1)/SOLVE_UNIT:split;
            hessian_pairs(S,sc,rec[ITEM_START],M,(warp+NW*(int)(entry&63u))*32,NW*parts*32,sv,q,slots,sks,pass);
            __syncthreads();
            for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){
                const unsigned e=tmap[t];
                T v[3];
#pragma unroll
                for(int ch=0;ch<3;++ch){T a=T(0);
#pragma unroll
                    for(int w2=0;w2<NW;++w2){T* p=&tile_of(w2)[ch][e>>11];a+=*p;*p=T(0);}
                    v[ch]=a;}
                add_tile_node(S,rec,e,v[0],v[1],v[2]);}}
        const double s=warp_value(sks);
        if(lane==0) part[warp][0]=s;};
    // warp 0: the CTA's sums into the slot of this phase, a sum per lane
    auto contribute=[&](int ns,bool with_max){
        SolveSlot& o=ctr->solve[phase&3];
        if(lane<ns){
            double v=0.;
#pragma unroll
            for(int w=0;w<NW;++w) v+=part[w][lane];
            if(v!=0.) atomicAdd(&o.sum[lane],v);}
        if(lane==3&&with_max){double m=0.;for(int w=0;w<NW;++w) m=fmax(m,part[w][3]);if(m>0.) atomicMax(&o.max0,dbits(m));}};
    // the slot two phases on: its readers have all arrived at the barrier before this one
    auto clear_ahead=[&]{
        if(blockIdx.x==0){SolveSlot& o=ctr->solve[(phase+2)&3];o.sum[0]=o.sum[1]=o.sum[2]=0.;o.max0=0ull;}};
    auto read_slot=[&](double (&s)[3],double& mx){
        const volatile SolveSlot& o=ctr->solve[phase&3];
        s[0]=o.sum[0];s[1]=o.sum[1];s[2]=o.sum[2];mx=bitsd(o.max0);};
    const double eps=1.1920928955078125e-07;     // FP32, as k_cg_start and k_cg_update
    // x = v*: r = b - A x and the first check
    product(true,T(0));
    if(!solve_barrier(ctr,arrived(),[]{},clear_ahead,[]{})) return;
    ++phase;
    {   NodeSum<T> rr;T amax=T(0);
        for(int blk=b0;blk<b1;++blk) cg_start_block(S,blk,ps.kdt,rr,amax);
        const double a=warp_value(rr),m=(double)warp_max<T>(amax);
        if(lane==0){part[warp][0]=a;part[warp][3]=m;}}
    double rho=0.,msq=0.,rmax=0.,beta=0.,rs_sum=0.,ss_sum=0.;        // thread 0 of every CTA: equal values
    int iters=0,converged=0;
    const double tol=S.cg[0].tol,tol2=tol*tol;
    // sqrt(mx) <= tol; the root (on the barriers' critical path) only where rounding could decide
    auto small=[&](double mx){return tol<0.?false:mx<tol2*(1.-1e-14)?true:mx>tol2*(1.+1e-14)?false:sqrt(mx)<=tol;};
    if(!solve_barrier(ctr,arrived(),[&]{contribute(1,true);},clear_ahead,[&]{
        double s[3],mx;read_slot(s,mx);
        rmax=mx;rho=msq=s[0];
        converged=small(mx)&&(0>=sc.cg_min_iters||sqrt(mx)<eps);
        sh_stop=converged||sc.cg_max_iters<=0||max_trips<=0;sh_beta=T(0);})) return;
    while(!sh_stop){
        ++phase;
        const T be=sh_beta;
        product(false,be);
        if(!solve_barrier(ctr,arrived(),[&]{contribute(1,false);},[&]{
            clear_ahead();
            if(iters>0) msq=rho+beta*(2.*rs_sum+beta*ss_sum);},[&]{
            double s[3],mx;read_slot(s,mx);
            const double sq=(double)ps.sks*s[0]+msq;
            sh_alpha=(T)(sq!=0.?rho/sq:(double)FLT_MAX);})) return;
        ++phase;
        {   const T alpha=sh_alpha;
            NodeSum<T> rr,rs,ss;T amax=T(0);
            for(int blk=b0;blk<b1;++blk) cg_update_block(S,((long long)blk<<6),alpha,be,ps.kdt,rr,rs,ss,amax);
            const double a=warp_value(rr),b=warp_value(rs),c=warp_value(ss),m=(double)warp_max<T>(amax);
            if(lane==0){part[warp][0]=a;part[warp][1]=b;part[warp][2]=c;part[warp][3]=m;}}
        if(!solve_barrier(ctr,arrived(),[&]{contribute(3,true);},clear_ahead,[&]{
            double s[3],mx;read_slot(s,mx);
            ++iters;rmax=mx;
            converged=small(mx)&&(iters>=sc.cg_min_iters||sqrt(mx)<eps);
            beta=s[0]/rho;rho=s[0];rs_sum=s[1];ss_sum=s[2];
            sh_beta=(T)beta;sh_stop=converged||iters>=sc.cg_max_iters||iters>=max_trips;})) return;}
    if(blockIdx.x==0&&threadIdx.x==0){
        CGState& st=S.cg[0];
        st.rho=rho;st.beta=beta;st.msq=msq;st.residual=sqrt(rmax);st.iters=iters;st.done=1;st.converged=converged;
        if(!converged) atomicOr(&ctr->error,ERR_CG_NOT_CONVERGED);
        ctr->any_active=0;ctr->loop_iters=iters;ctr->total_trips+=iters;}
}

// =====================================================================================
// K7: G2P (Update_Particle_Velocities_And_Positions, MPM_Example.cpp:633-660): for nodes
// with w>0, V_pic = sum w v*, V_flip = V + sum w (v*-v), grad v = sum v* grad w^T;
// Fe += dt grad v Fe; V = flip V_flip + (1-flip) V_pic; X += dt V_pic; particles outside
// [dx/2, 1-dx/2]^3 are removed.
// =====================================================================================
template<class T,int MINB> __global__ void __launch_bounds__(XFER_THREADS,MINB) k_g2p(DevState<T> S)
{
    pdl_enter();
    __shared__ T tv[6][TILE_S];
    __shared__ int nbr[27];
    const unsigned nc=min(S.ctr->n_chunks,(unsigned)S.chunk_cap),nv=S.ctr->n_valid;
    for(long long c=blockIdx.x;c<nc;c+=gridDim.x){
        ChunkInfo<T> ci;load_chunk(S,c,nc,nv,ci,nbr);
        __syncthreads();
        for(int t=threadIdx.x;t<TILE_N;t+=blockDim.x){
            const long long node=tile_node(nbr,t);
            const int ta=tile_addr(t);
            if(node>=0){const V4<T> v=S.gv[node],x=S.gx[node];
                tv[0][ta]=v.x;tv[1][ta]=v.y;tv[2][ta]=v.z;tv[3][ta]=x.x;tv[4][ta]=x.y;tv[5][ta]=x.z;}
            else{for(int k=0;k<6;++k) tv[k][ta]=T(0);}}
        if(c+gridDim.x<nc){                 // the first particles of this CTA's next work item into L2
            const long long in=S.chunk_start[c+gridDim.x]+(long long)threadIdx.x;
            if(in<(long long)nv){
                auto pf=[](const void* p){asm volatile("prefetch.global.L2 [%0];"::"l"(p));};
#pragma unroll
                for(int k=0;k<15;++k) pf(S.pcur+(FX+k)*S.pcap+in);
                pf(S.keys+in);}}
        __syncthreads();
        const SceneDev<T>& sc=S.scenes[ci.scene];
        for(int i=ci.s+threadIdx.x;i<ci.e;i+=blockDim.x){
            const long long pc=S.pcap;
            if(i+(int)blockDim.x<ci.e){     // the thread's next particle into L2 (latency-bound on these loads)
                const int in=i+(int)blockDim.x;
                auto pf=[](const void* p){asm volatile("prefetch.global.L2 [%0];"::"l"(p));};
#pragma unroll
                for(int k=0;k<15;++k) pf(S.pcur+(FX+k)*pc+in);    // X, V, Fe
                pf(S.keys+in);}
            T X[3],V[3],F[9];
#pragma unroll
            for(int a=0;a<3;++a){X[a]=S.pcur[(FX+a)*pc+i];V[a]=S.pcur[(FV+a)*pc+i];}
#pragma unroll
            for(int k=0;k<9;++k) F[k]=S.pcur[(FF+k)*pc+i];
            Stencil<T> st;make_stencil(sc,ci.b,S.keys[i],X,st);
            // V_pic = sum w v*, the FLIP increment sum w (v* - v), grad v = sum v* grad w^T, contracted over z
            // first. Nodes with w = 0 (a particle exactly on a stencil edge) add nothing: their
            // weight and, along the same axis, the weight's derivative vanish together.
            T vp[3]={T(0),T(0),T(0)},vd[3]={T(0),T(0),T(0)};
            T G[9]={T(0),T(0),T(0),T(0),T(0),T(0),T(0),T(0),T(0)};
            const int tb=tile_addr(st.r[0]-1,st.r[1]-1,st.r[2]-1);
            if constexpr(sizeof(T)==4){
                // components 0 and 1 as packed pairs, component 2 scalar: each lane of a pair
                // is the same fused multiply-add (or subtraction) as the scalar form
                float2 vp01=make_float2(0.f,0.f),vd01=vp01,g0=vp01,g1=vp01,g2=vp01;   // g0 = (G[0], G[3]) ...
#pragma unroll
                for(int ox=0;ox<3;++ox)
#pragma unroll
                for(int oy=0;oy<3;++oy){
                    float2 ts01=make_float2(0.f,0.f),us01=ts01,to01=ts01;
                    float ts2=0.f,us2=0.f,to2=0.f;
#pragma unroll
                    for(int oz=0;oz<3;++oz){
                        const float wz=st.w[2][oz],dz=st.dw[2][oz];
                        const int t=tb+tile_addr(ox,oy,oz);
                        const float2 s01=make_float2(tv[3][t],tv[4][t]);
                        const float2 d01=__fadd2_rn(s01,make_float2(-tv[0][t],-tv[1][t]));
                        ts01=pfma(pdup(wz),s01,ts01);us01=pfma(pdup(dz),s01,us01);to01=pfma(pdup(wz),d01,to01);
                        const float s2=tv[5][t];
                        ts2=fmaf(wz,s2,ts2);us2=fmaf(dz,s2,us2);to2=fmaf(wz,s2-tv[2][t],to2);}
                    const float dxy=st.dw[0][ox]*st.w[1][oy],xdy=st.w[0][ox]*st.dw[1][oy],wxy=st.w[0][ox]*st.w[1][oy];
                    vp01=pfma(pdup(wxy),ts01,vp01);vd01=pfma(pdup(wxy),to01,vd01);
                    g0=pfma(pdup(dxy),ts01,g0);g1=pfma(pdup(xdy),ts01,g1);g2=pfma(pdup(wxy),us01,g2);
                    vp[2]=fmaf(wxy,ts2,vp[2]);vd[2]=fmaf(wxy,to2,vd[2]);
                    G[6]=fmaf(dxy,ts2,G[6]);G[7]=fmaf(xdy,ts2,G[7]);G[8]=fmaf(wxy,us2,G[8]);}
                vp[0]=vp01.x;vp[1]=vp01.y;vd[0]=vd01.x;vd[1]=vd01.y;
                G[0]=g0.x;G[3]=g0.y;G[1]=g1.x;G[4]=g1.y;G[2]=g2.x;G[5]=g2.y;}
            else{
#pragma unroll
            for(int ox=0;ox<3;++ox)
#pragma unroll
            for(int oy=0;oy<3;++oy){
                T ts[3]={T(0),T(0),T(0)},us[3]={T(0),T(0),T(0)},to[3]={T(0),T(0),T(0)};
#pragma unroll
                for(int oz=0;oz<3;++oz){
                    const T wz=st.w[2][oz],dz=st.dw[2][oz];
                    const int t=tb+tile_addr(ox,oy,oz);
#pragma unroll
                    for(int a=0;a<3;++a){const T sa=tv[3+a][t];ts[a]+=wz*sa;us[a]+=dz*sa;to[a]+=wz*(sa-tv[a][t]);}}
                const T dxy=st.dw[0][ox]*st.w[1][oy],xdy=st.w[0][ox]*st.dw[1][oy],wxy=st.w[0][ox]*st.w[1][oy];
#pragma unroll
                for(int a=0;a<3;++a){
                    vp[a]+=wxy*ts[a];vd[a]+=wxy*to[a];
                    G[3*a]+=dxy*ts[a];G[3*a+1]+=xdy*ts[a];G[3*a+2]+=wxy*us[a];}}}
            T vf[3];
#pragma unroll
            for(int a=0;a<3;++a) vf[a]=V[a]+vd[a];
            const T dt=(T)(*S.dtp);
            if(sc.eos){
                // EOS fluid: density /= 1 + dt tr(grad v), Fe untouched (MPM_Example.cpp:646)
                const T rho=S.pcur[FJP*pc+i];
                S.pcur[FJP*pc+i]=rho/(T(1)+dt*(G[0]+G[4]+G[8]));}
            else{
                T GF[9];mat_mul(G,F,GF);
#pragma unroll
                for(int k=0;k<9;++k) S.pcur[(FF+k)*pc+i]=F[k]+dt*GF[k];}
            const T flip=sc.flip;
            bool inside=true,fin=true;
#pragma unroll
            for(int a=0;a<3;++a){
                const T vn=vf[a]*flip+vp[a]*(T(1)-flip);
                const T xn=X[a]+vp[a]*dt;
                S.pcur[(FV+a)*pc+i]=vn;S.pcur[(FX+a)*pc+i]=xn;
                if(!isfinite(xn)) fin=false;
                const T lo=T(0)+T(0.5)*sc.dx[a],hi=T(1)-T(0.5)*sc.dx[a];
                if(!(xn>=lo&&xn<=hi)) inside=false;}
            if(!fin){atomicOr(&S.ctr->error,ERR_NONFINITE);atomicMax(&S.ctr->bad_scene1,(unsigned)ci.scene+1u);}
            if(!inside) S.scn_cur[i]=-(ci.scene+1);
        }
        __syncthreads();
    }
}

// =====================================================================================
// K8: the substep size of mpm_advance_to_time (MPM_Driver::Advance_To_Target_Time,
// MPM_Driver.cpp:55-80). Per scene, max_v over its valid particles (Max_Particle_Velocity,
// MPM_Example.cpp:375-387) gives dt_s = clamp(cfl dx / max(max_v, 1e-2), dt_min, dt_max);
// the substep takes the smallest dt_s of the batch (one substep sequence for all scenes;
// with one scene this is the reference's rule). Then the end-of-frame split: the last
// substep lands exactly on the target, and the one before it halves the rest when less
// than two steps remain. The last CTA writes dt, advances the clock and sets `h_more`
// (when given) to whether another substep follows.
// =====================================================================================
template<class T> __global__ void __launch_bounds__(NODE_THREADS) k_cfl(DevState<T> S,FrameState* F,double* dt_out,unsigned long long h_more,int use_more)
{
    __shared__ SceneRed R;
    __shared__ unsigned long long dtbits;
    const unsigned parts=taking_part(S.n_total,blockDim.x);
    if(blockIdx.x>=parts) return;
    red_init(R,S.n_scenes);
    if(threadIdx.x==0) dtbits=dbits(F->dt_max);
    __syncthreads();
    const long long pc=S.pcap;
    for(long long i=blockIdx.x*(long long)blockDim.x+threadIdx.x;i<S.n_total;i+=(long long)gridDim.x*blockDim.x){
        const int s=S.scn_cur[i];
        if(s<0) continue;
        T a=T(0);
#pragma unroll
        for(int k=0;k<3;++k){const T v=S.pcur[(FV+k)*pc+i];a+=v*v;}
        const double v2=(double)a;
        if(v2>0.) atomicMax(&R.mx[s],dbits(v2));}
    const bool last=red_finish<false>(R,S.n_scenes,S.acc2,&S.ctr->ticket[4],parts,[&](int i,double mx,unsigned long long){
        const double vmax=sqrt(mx);
        const double dt=fmax(F->dt_min,fmin(F->dt_max,F->cfl*(double)S.scenes[i].dx[0]/fmax(vmax,1e-2)));
        atomicMin(&dtbits,dbits(dt));
    });
    if(last&&threadIdx.x==0){
        double dt=bitsd(dtbits);
        const double rem=F->target-F->time;
        int done=0;
        if(rem<dt*1.001){dt=rem;done=1;}
        else if(rem<2.*dt) dt=rem*0.5;
        F->substeps+=1;
        if(F->substeps>=F->max_substeps) done=1;
        F->time=(done&&dt==rem)?F->target:F->time+dt;
        F->dt_last=dt;F->done=done;
        *dt_out=dt;
        if(use_more) cudaGraphSetConditional((cudaGraphConditionalHandle)h_more,done?0u:1u);}
}
// Loop condition of the frame graph: continue while the latest substep did not end it.
static __global__ void k_frame_cond(const FrameState* F,unsigned long long h)
{
    if(threadIdx.x==0&&blockIdx.x==0) cudaGraphSetConditional((cudaGraphConditionalHandle)h,F->done?0u:1u);
}

} // namespace mpm
