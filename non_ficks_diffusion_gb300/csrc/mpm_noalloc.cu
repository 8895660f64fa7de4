// mpm_noalloc.cu — the stable radix sort of (cell key, index) pairs, callable without any
// device allocation.
//
// Some callers cannot allocate device memory at the point where they sort: a host that
// records its frame loop into a CUDA graph (cudaMalloc is not allowed while a stream is
// being captured), a real-time loop that must not take cudaMalloc's implicit device
// synchronisation, or an embedding framework that owns all device memory through its own
// allocator. They pass their key and value arrays in device memory; the sort's working
// memory (ping-pong buffers, digit histograms, per-tile status words) comes from the fixed
// static device array below, reserved when the library is loaded on a GPU and held until
// the process exits.
#include "mpm_gb300.h"
#include "mpm_binning.cuh"

#include <cuda.h>   // CUcontext and CUresult only: the two driver functions are looked up through the runtime

#include <algorithm>
#include <mutex>

using namespace mpm;

namespace {

constexpr long long kMaxPairs=MPM_NOALLOC_SORT_MAX;
// Keys per thread of a tile. A pass takes as long as one tile's chain of steps and the
// look-back over all tiles, so small sorts want short tiles and large ones fewer: three passes
// of 5K random pairs take 23 us with 4 keys a thread, 35 with 8, 43 with 16; of 300K 37, 43
// and 62; of 500K 45, 47 and 64; of 10^6 68, 59 and 67.
constexpr int NS_THREADS=512, NS_WARPS=NS_THREADS/32, NS_LOOKBACK=16;
constexpr long long NS_SMALL=500000;
constexpr int ns_items(long long n){return n<=NS_SMALL?4:8;}
constexpr int ns_smem(int items){return NS_THREADS*items*8;}
constexpr long long kMaxTiles=256;
static_assert((NS_SMALL+NS_THREADS*4-1)/(NS_THREADS*4)<=kMaxTiles&&(kMaxPairs+NS_THREADS*8-1)/(NS_THREADS*8)<=kMaxTiles,"status words");

// One static scratch area per device: ping-pong keys and values; what a call zeroes first:
// tile counters, digit histograms of all passes, and the passes' status words.
struct NoallocScratch {
    unsigned keys[kMaxPairs];
    int vals[kMaxPairs];
    unsigned counter[4];
    unsigned hist[4][256];
    unsigned status[4*kMaxTiles*256];
};
static __device__ __align__(256) NoallocScratch g_noalloc_scratch;

// Device address of the scratch. In host code the symbol itself is only a host-side
// stand-in; its device address comes from cudaGetSymbolAddress with the device current.
// That address belongs to the module loaded in the current context, so it is cached per
// device together with the identity of the context it was looked up in (cuCtxGetId: unique
// for the life of the process). A context created anew on the device (after
// cudaDeviceReset, or the primary context released and retained again) gets a new identity
// and the address is looked up again.
typedef CUresult (*FnCtxGetCurrent)(CUcontext*);
typedef CUresult (*FnCtxGetId)(CUcontext,unsigned long long*);
struct CachedScratch { unsigned long long ctx_id; NoallocScratch* ptr; };

std::mutex g_mutex;
CachedScratch g_cache[64]={};
FnCtxGetCurrent g_ctx_get_current=nullptr;
FnCtxGetId g_ctx_get_id=nullptr;

// Identity of the calling thread's current context; 0 when none is current.
bool current_context_id(unsigned long long* id)
{
    if(!g_ctx_get_current||!g_ctx_get_id){
        void* f1=nullptr;void* f2=nullptr;cudaDriverEntryPointQueryResult q1,q2;
        if(cudaGetDriverEntryPointByVersion("cuCtxGetCurrent",&f1,12000,cudaEnableDefault,&q1)!=cudaSuccess||
           cudaGetDriverEntryPointByVersion("cuCtxGetId",&f2,12000,cudaEnableDefault,&q2)!=cudaSuccess||
           q1!=cudaDriverEntryPointSuccess||q2!=cudaDriverEntryPointSuccess||!f1||!f2) return false;
        g_ctx_get_current=(FnCtxGetCurrent)f1;g_ctx_get_id=(FnCtxGetId)f2;}
    CUcontext ctx=nullptr;
    if(g_ctx_get_current(&ctx)!=CUDA_SUCCESS) return false;
    *id=0;
    if(!ctx) return true;
    return g_ctx_get_id(ctx,id)==CUDA_SUCCESS;
}

template<int ITEMS> __global__ void k_sort_pass(const unsigned*,const int*,unsigned*,int*,long long,int,const unsigned*,unsigned*,unsigned*,int,int,bool);
NoallocScratch* scratch_for(int dev)
{
    std::lock_guard<std::mutex> lock(g_mutex);
    if(dev<0||dev>=64) return nullptr;
    unsigned long long id=0;
    if(!current_context_id(&id)) return nullptr;
    if(id!=0&&g_cache[dev].ptr&&g_cache[dev].ctx_id==id) return g_cache[dev].ptr;
    void* p=nullptr;
    if(cudaGetSymbolAddress(&p,g_noalloc_scratch)!=cudaSuccess) return nullptr;   // makes the device's context current
    if(!current_context_id(&id)||id==0) return nullptr;
    // the larger tile needs more dynamic shared memory than a kernel gets by default
    if(cudaFuncSetAttribute(k_sort_pass<8>,cudaFuncAttributeMaxDynamicSharedMemorySize,ns_smem(8))!=cudaSuccess) return nullptr;
    g_cache[dev].ctx_id=id;g_cache[dev].ptr=(NoallocScratch*)p;
    return g_cache[dev].ptr;
}

// Launches one kernel and returns that launch's own status (an error left behind by
// earlier, unrelated work in the process is neither reported nor cleared here).
template<class... KA,class... A> cudaError_t launch(void(*k)(KA...),int grid,int block,int smem,cudaStream_t st,A&&... a)
{
    cudaLaunchConfig_t cfg={};
    cfg.gridDim=dim3((unsigned)grid);cfg.blockDim=dim3((unsigned)block);cfg.dynamicSmemBytes=smem;cfg.stream=st;
    cudaLaunchAttribute at[1];               // scheduled while the kernel before drains (pdl_enter waits for it)
    at[0].id=cudaLaunchAttributeProgrammaticStreamSerialization;at[0].val.programmaticStreamSerializationAllowed=1;
    cfg.attrs=at;cfg.numAttrs=1;
    return cudaLaunchKernelEx(&cfg,k,std::forward<A>(a)...);
}

// Digit histograms of all passes in one reading of the keys.
__global__ void __launch_bounds__(512) k_sort_hist(const unsigned* __restrict__ keys,long long n,int shift,int passes,unsigned* hist)
{
    pdl_enter();
    __shared__ unsigned h[4][256];
    for(int t=threadIdx.x;t<4*256;t+=blockDim.x) (&h[0][0])[t]=0;
    __syncthreads();
    for(long long i=blockIdx.x*(long long)blockDim.x+threadIdx.x;i<n;i+=(long long)gridDim.x*blockDim.x){
        const unsigned k=keys[i];
        for(int p=0;p<passes;++p) atomicAdd(&h[p][(k>>(shift+8*p))&255u],1u);}
    __syncthreads();
    for(int t=threadIdx.x;t<passes*256;t+=blockDim.x){const unsigned v=(&h[0][0])[t];if(v) atomicAdd(&hist[t],v);}
}
// One stable 8-bit pass: the tiles of k_onesweep (ticket order, decoupled look-back) for keys in
// any order. A wait for an earlier tile's word gives up after `spin_limit` polls; the thread
// then counts its digit itself, in the keys of that tile and of all before it, so that the result
// does not depend on the waits. (`publish` false, for the check of that path: no words are
// published.) Peers come from eight ballots instead of match.any, whose cost
// grows with the distinct digits of a warp, and the tile's pairs go through shared memory
// in digit order, so that each digit's run is stored contiguously. A pass of 10^6 random
// pairs takes about 17 us, against 44 for five kernels (histogram, three of a scan, scatter).
// Bound by latency: its 16 MB of traffic take 2.4 us.
template<int ITEMS> __global__ void __launch_bounds__(NS_THREADS) k_sort_pass(const unsigned* __restrict__ kin,const int* __restrict__ vin,
    unsigned* __restrict__ kout,int* __restrict__ vout,long long n,int shift,const unsigned* __restrict__ hist,unsigned* status,
    unsigned* tile_counter,int num_tiles,int spin_limit,bool publish)
{
    pdl_enter();
    extern __shared__ unsigned smem[];
    unsigned* skey=smem;int* sval=(int*)(smem+NS_THREADS*ITEMS);
    __shared__ unsigned wcnt[NS_WARPS][256];
    __shared__ unsigned first[256],out0[256],wsum[NS_WARPS];
    __shared__ int tile_sh;
    const int tid=threadIdx.x,w=tid>>5,lane=tid&31;
    // exclusive scan over the 256 digits, one per thread below 256 (every thread calls)
    auto scan256=[&](unsigned v){
        unsigned x=v;
#pragma unroll
        for(int o=1;o<32;o<<=1){const unsigned y=__shfl_up_sync(0xffffffffu,x,o);if(lane>=o) x+=y;}
        if(lane==31) wsum[w]=x;
        __syncthreads();
        unsigned b=0;
        for(int q=0;q<w&&q<8;++q) b+=wsum[q];
        __syncthreads();
        return b+x-v;};
    const unsigned digit0=scan256(tid<256?hist[tid]:0u);      // where digit tid starts
    for(;;){
        if(tid==0) tile_sh=(int)atomicAdd(tile_counter,1u);
        for(int t=tid;t<NS_WARPS*256;t+=NS_THREADS) (&wcnt[0][0])[t]=0;
        __syncthreads();
        const int tile=tile_sh;
        if(tile>=num_tiles) break;                             // uniform
        const long long t0=(long long)tile*NS_THREADS*ITEMS,base=t0+(long long)w*(ITEMS*32);
        unsigned k[ITEMS];unsigned short r[ITEMS];
#pragma unroll
        for(int j=0;j<ITEMS;++j){const long long i=base+j*32+lane;k[j]=i<n?kin[i]:0u;}
#pragma unroll
        for(int j=0;j<ITEMS;++j){
            const bool valid=base+j*32+lane<n;
            const unsigned d=(k[j]>>shift)&255u;
            unsigned peers=__ballot_sync(0xffffffffu,valid);
#pragma unroll
            for(int b=0;b<8;++b){const bool bit=(d>>b)&1u;const unsigned m=__ballot_sync(0xffffffffu,bit);peers&=bit?m:~m;}
            const unsigned rank=__popc(peers&lanemask_lt()),before=valid?wcnt[w][d]:0u;
            __syncwarp();
            if(valid&&rank==0) wcnt[w][d]=before+__popc(peers);
            __syncwarp();
            r[j]=(unsigned short)(before+rank);}
        __syncthreads();
        unsigned count=0;
        if(tid<256){
#pragma unroll
            for(int q=0;q<NS_WARPS;++q){const unsigned c=wcnt[q][tid];wcnt[q][tid]=count;count+=c;}
            if(publish) atomicExch(status+(long long)tile*256+tid,(tile==0?OS_PRE:OS_AGG)|count);}
        const unsigned f=scan256(count);
        if(tid<256) first[tid]=f;
        __syncthreads();
#pragma unroll
        for(int j=0;j<ITEMS;++j){
            const long long i=base+j*32+lane;
            if(i<n){
                const unsigned d=(k[j]>>shift)&255u,at=first[d]+wcnt[w][d]+r[j];
                skey[at]=k[j];sval[at]=vin?vin[i]:(int)i;}}
        if(tid<256){
            unsigned excl=0;
            if(tile>0){
                bool done=false;
                long long counted=0;              // keys from the first on that this thread has to count
                for(int t=tile-1;t>=0&&!done;t-=NS_LOOKBACK){
                    unsigned v[NS_LOOKBACK];
#pragma unroll
                    for(int u=0;u<NS_LOOKBACK;++u) v[u]=t-u>=0?os_load(status+(long long)(t-u)*256+tid):OS_PRE;
#pragma unroll
                    for(int u=0;u<NS_LOOKBACK;++u){
                        if(done||t-u<0) continue;
                        unsigned x=v[u];
                        for(int spins=0;(x&~OS_MASK)==0u&&spins<spin_limit;++spins){__nanosleep(32);x=os_load(status+(long long)(t-u)*256+tid);}
                        if((x&~OS_MASK)==0u){counted=(long long)(t-u+1)*NS_THREADS*ITEMS;done=true;break;}
                        excl+=x&OS_MASK;
                        if((x&~OS_MASK)!=OS_AGG) done=true;}}
                for(long long i=0;i<counted;++i) excl+=((kin[i]>>shift)&255u)==(unsigned)tid;
                if(publish) atomicExch(status+(long long)tile*256+tid,OS_PRE|(excl+count));}
            out0[tid]=digit0+excl-f;}
        __syncthreads();
        const int m=(int)(n-t0<NS_THREADS*ITEMS?n-t0:NS_THREADS*ITEMS);
        for(int i=tid;i<m;i+=NS_THREADS){
            const unsigned key=skey[i],pos=out0[(key>>shift)&255u]+i;
            // always, unless calls overlap and mix their counts: that spoils their results, not other memory
            if(pos<n){kout[pos]=key;vout[pos]=sval[i];}}
        __syncthreads();
    }
}

mpm_status sort_pairs(const uint32_t* keys_in,const int32_t* vals_in,uint32_t* keys_out,int32_t* vals_out,
                      long long n,int begin_bit,int end_bit,void* stream,int spin_limit,bool publish)
{
    if(n<0||n>kMaxPairs||!keys_out||!vals_out||(n>0&&!keys_in)) return MPM_BAD_ARG;
    if(begin_bit<0||end_bit>32||begin_bit>=end_bit) return MPM_BAD_ARG;
    if((const void*)keys_in==(const void*)keys_out||(vals_in&&(const void*)vals_in==(const void*)vals_out)) return MPM_BAD_ARG;
    if(n==0) return MPM_OK;
    int dev=0;
    if(cudaGetDevice(&dev)!=cudaSuccess) return MPM_CUDA_ERROR;
    NoallocScratch* sc=scratch_for(dev);
    if(!sc) return MPM_CUDA_ERROR;
    cudaStream_t st=(cudaStream_t)stream;
    int num_sms=0;
    if(cudaDeviceGetAttribute(&num_sms,cudaDevAttrMultiProcessorCount,dev)!=cudaSuccess) return MPM_CUDA_ERROR;
    const int passes=(end_bit-begin_bit+7)/8,items=ns_items(n);
    const int num_tiles=(int)((n+(long long)NS_THREADS*items-1)/((long long)NS_THREADS*items));
    const int g=std::min(num_tiles,2*num_sms);
    // the counters, histograms and used status words of all passes lie side by side
    const size_t zero=(char*)sc->status-(char*)sc->counter+sizeof(unsigned)*256*(size_t)num_tiles*passes;
    if(cudaMemsetAsync(sc->counter,0,zero,st)!=cudaSuccess) return MPM_CUDA_ERROR;
    if(launch(k_sort_hist,(int)std::min<long long>((n+2047)/2048,2LL*num_sms),512,0,st,keys_in,n,begin_bit,passes,&sc->hist[0][0])!=cudaSuccess)
        return MPM_CUDA_ERROR;
    // Pass p writes to the caller's output when (passes-1-p) is even, so the last pass
    // always lands there; the other passes use the static ping-pong buffers.
    const unsigned* kin=keys_in;const int* vin=vals_in;
    for(int p=0;p<passes;++p){
        const bool to_out=((passes-1-p)%2)==0;
        unsigned* kout=to_out?keys_out:sc->keys;int* vout=to_out?vals_out:sc->vals;
        const unsigned* h=sc->hist[p];unsigned* status=sc->status+(long long)p*num_tiles*256;
        auto pass=[&](auto kernel){
            return launch(kernel,g,NS_THREADS,ns_smem(items),st,kin,vin,kout,vout,n,begin_bit+8*p,h,status,sc->counter+p,num_tiles,spin_limit,publish);};
        const cudaError_t e=items==4?pass(k_sort_pass<4>):pass(k_sort_pass<8>);
        if(e!=cudaSuccess) return MPM_CUDA_ERROR;
        kin=kout;vin=vout;}
    return MPM_OK;
}

} // namespace

// Polls of about 40 ns each before a look-back counts for itself: a few milliseconds, against the
// microseconds in which a resident CTA publishes.
constexpr int kSortSpinLimit=1<<16;

extern "C" mpm_status mpm_sort_pairs_noalloc(const uint32_t* keys_in,const int32_t* vals_in,uint32_t* keys_out,int32_t* vals_out,
                                             long long n,int begin_bit,int end_bit,void* stream)
{
    return sort_pairs(keys_in,vals_in,keys_out,vals_out,n,begin_bit,end_bit,stream,kSortSpinLimit,true);
}
extern "C" mpm_status mpm_selftest_sort_wait(const uint32_t* keys_in,const int32_t* vals_in,uint32_t* keys_out,int32_t* vals_out,
                                             long long n,int begin_bit,int end_bit,int spin_limit,void* stream)
{
    if(spin_limit<1||spin_limit>1000) return MPM_BAD_ARG;
    return sort_pairs(keys_in,vals_in,keys_out,vals_out,n,begin_bit,end_bit,stream,spin_limit,false);
}
